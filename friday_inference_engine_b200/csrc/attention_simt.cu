// Causal grouped-query attention over the paged cache, CUDA cores, fp32 arithmetic.
//
// One kernel serves prompts and decoding, fp32 and bf16 storage, every head size up
// to 256 (any multiple of 2), any number of heads and groups, full and windowed
// layers, windows that keep a sequence's first keys in sight, and values whose size
// differs from the keys'.  A warp owns one (query row, head, split): it walks its range of keys with
// an online softmax (running maximum m, sum l, weighted values o), the head's
// dimensions spread over the lanes.  With more than one split the warps write
// (m, l, o) to a scratch buffer and a second kernel merges them; that keeps many
// warps busy when a few rows face long contexts (decoding).
//
// It is the true 32-bit path's attention and the bf16 path's fallback.  Reference:
// decodeAttentionKernel and the split/combine pair (attention_kernels.cu:29-111,
// 131-235), prefillAttentionKernel (:513-645); mask by range as there (j <= position).
//
// Geometry of a step: every row carries its sequence (row_seq, an index into the step's
// block table) and its position (row_pos); it sees the keys of its sequence up to that
// position.  Keys and values of position j are in page block_table[seq][j / page], row
// j % page, of pools laid out [pages][page][nkv][hd] (keys) and [pages][page][nkv][vd] (values).
//
// With a window W and `keep_first` F, row i sees key j if j <= i and (i - j < W or j < F): the keys
// a warp walks are the kept ones below the window's start followed by the window's.
#include <math.h>

#include <atomic>

#include "attention_merge.cuh"
#include "common.cuh"

FR_EXPORT const char* attention_simt_last_error() { return fr_error_text; }

namespace {

constexpr int MOST_PER_LANE = 8;   // head sizes up to 256

struct AttnArgs {
    const void* q;        // [rows][q_stride] ; head h at h*hd
    void* out;            // [rows][nq*hd]
    const void* k_pool;
    const void* v_pool;
    const int* block_table;
    const int* row_seq;   // [rows] sequence of the row, < 0: padding row (output zeros)
    const int* row_pos;   // [rows] position of the row
    float* part;          // [rows][nq][splits][hd + 2] when splits > 1
    int table_width, page, rows, nq, nkv, hd, q_stride, window, splits;
    float scale;
    int vd, keep_first;   // size of a value head; keys below keep_first stay visible behind a window
    float out_scale;      // the result is multiplied by this
};

template <int N>
struct Number {
    static constexpr int value = N;
};

// MAX_PER_LANE: dimensions per lane; KEYS keys at a time, four where no more than four are left: their loads are issued together,
// keys before values (bf16 heads of 65 to 128: key by key, a tenth faster), so that a warp waits for memory once per round.  fp32, us, four at a time / as launched below: 28 heads of 32,
// 4 rows, a window of 24 keys 8.0 / 4.6; of 64, 333 rows 267 / 183, 8 rows x 4,000 keys 166 / 113; of 128, 333 rows 275 / 207.
template <typename T, int MAX_PER_LANE, int KEYS>
__global__ void __launch_bounds__(128) attention_kernel(AttnArgs p) {
    constexpr bool VALUES_LAST = sizeof(T) == 4 || MAX_PER_LANE != 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * 4 + warp;          // (row, head)
    if (item >= p.rows * p.nq) return;
    const int row = item / p.nq, h = item - row * p.nq;
    const int split = blockIdx.y;
    fr_pdl_wait();
    fr_pdl_launch();
    const int seq = p.row_seq[row];
    T* o_row = (T*)p.out + (size_t)row * p.nq * p.vd + (size_t)h * p.vd;
    float* part = p.splits > 1 ? p.part + ((size_t)item * p.splits + split) * (p.vd + 2) : nullptr;

    float qv[MAX_PER_LANE], acc[MAX_PER_LANE];
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;

    if (seq >= 0) {
        const int pos = p.row_pos[row];
        const int kvh = h / (p.nq / p.nkv);
        const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
        const int kept = min(p.keep_first, lo);         // kept keys below the window's start
        const int n = kept + pos - lo + 1;
        const int chunk = (n + p.splits - 1) / p.splits;
        const int i0 = split * chunk;
        const int i1 = min(i0 + chunk, n);
        const T* q = (const T*)p.q + (size_t)row * p.q_stride + (size_t)h * p.hd;
#pragma unroll
        for (int i = 0; i < MAX_PER_LANE; ++i) {
            const int d = lane + 32 * i;
            qv[i] = d < p.hd ? fr_load(q + d) * p.scale : 0.f;
        }
        const int* table = p.block_table + (size_t)seq * p.table_width;
        // this lane's share of a key's score; its value too where v is given
        auto dot = [&](const T* k, const T* v, float& score, float (&value)[MAX_PER_LANE]) {
            float s = 0.f;
#pragma unroll
            for (int c = 0; c < MAX_PER_LANE; ++c) {
                const int d = lane + 32 * c;
                if (d < p.hd) s = fmaf(qv[c], fr_load(k + d), s);
                if (!VALUES_LAST) value[c] = d < p.vd ? fr_load(v + d) : 0.f;
            }
            score = s;
        };
        auto round = [&](auto number, int i) {
            constexpr int N = decltype(number)::value;
            const T* kr[N];
            const T* vr[N];
            float sk[N], vv[N][MAX_PER_LANE];
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const int iu = min(i + u, i1 - 1);           // past the end: the last key again (its weight is set to zero)
                const int j = iu < kept ? iu : lo + (iu - kept);
                const size_t at = ((size_t)table[j / p.page] * p.page + j % p.page) * p.nkv + kvh;
                kr[u] = (const T*)p.k_pool + at * p.hd;
                vr[u] = (const T*)p.v_pool + at * p.vd;
                if (!VALUES_LAST) dot(kr[u], vr[u], sk[u], vv[u]);
            }
            if (VALUES_LAST) {
#pragma unroll
                for (int u = 0; u < N; ++u) dot(kr[u], nullptr, sk[u], vv[u]);
#pragma unroll
                for (int u = 0; u < N; ++u)
#pragma unroll
                    for (int c = 0; c < MAX_PER_LANE; ++c) {
                        const int d = lane + 32 * c;
                        vv[u][c] = d < p.vd ? fr_load(vr[u] + d) : 0.f;
                    }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < N; ++u) sk[u] += __shfl_xor_sync(0xffffffffu, sk[u], o);
            float m_new = m;
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (i + u < i1) m_new = fmaxf(m_new, sk[u]);
            const float alpha = expf(m - m_new);      // exp(-inf) = 0 on the first keys
            float e[N], sum = 0.f;
#pragma unroll
            for (int u = 0; u < N; ++u) {
                e[u] = i + u < i1 ? expf(sk[u] - m_new) : 0.f;
                sum += e[u];
            }
            l = l * alpha + sum;
#pragma unroll
            for (int c = 0; c < MAX_PER_LANE; ++c) {
                // (large heads: the sums under the condition of their loads, which the compiler then keeps together; without it
                // heads of 192 and 256 took half as long again, with it smaller ones a tenth longer)
                if (MAX_PER_LANE < 8 || lane + 32 * c < p.vd) {
                    float add = 0.f;
#pragma unroll
                    for (int u = 0; u < N; ++u) add = fmaf(e[u], vv[u][c], add);
                    acc[c] = acc[c] * alpha + add;
                }
            }
            m = m_new;
        };
        int i = i0;
        if (KEYS > 4)
            for (; i1 - i > 4; i += KEYS) round(Number<KEYS>{}, i);
        for (; i < i1; i += 4) round(Number<4>{}, i);
    }
    if (part == nullptr) {
        const float inv = l > 0.f ? p.out_scale / l : 0.f;
#pragma unroll
        for (int i = 0; i < MAX_PER_LANE; ++i) {
            const int d = lane + 32 * i;
            if (d < p.vd) fr_store(o_row + d, acc[i] * inv);
        }
    } else {
#pragma unroll
        for (int i = 0; i < MAX_PER_LANE; ++i) {
            const int d = lane + 32 * i;
            if (d < p.vd) part[d] = acc[i];
        }
        if (lane == 0) {
            part[p.vd] = m;
            part[p.vd + 1] = l;
        }
    }
}

// Prompts in fp32.  The kernel above reads every key and value for every query row; here a block takes 16 RPT rows, the query
// heads of one kv head for as many consecutive tokens as that makes, and walks 32 keys at a time, which pass through shared memory once
// for all of them.  128 threads: a thread has RPT rows' scores with four keys, then the same rows' results in HD / 8
// channels, so that a row's scores, maximum and weights stay within a warp.  Scores are summed 16 dimensions at a time, which keeps
// their error that of the sums over lanes above.  Bound by the multiply-adds (each needs an eighth of a 16-byte read from shared
// memory with four rows per thread) where blocks are many; two rows per thread where they are few.  One prompt of 333 rows, 28 query and 4 kv heads of 128: 180 us with the
// kernel above, 90 with 64 rows a block, 64 with 32.
constexpr int PT_KEYS = 32, PT_THREADS = 128, PT_MOST_ROWS = 64;

struct PromptArgs {
    const float* q;
    float* out;
    const float* k_pool;
    const float* v_pool;
    const int* block_table;
    const int* row_seq;
    const int* seq_start;
    const int* seq_qlen;
    const int* seq_pos0;
    int table_width, page, nq, nkv, hd, q_stride, window;
    float scale;
};
template <int HD, int RPT>
constexpr int prompt_smem() { return (16 * RPT * (HD + 4) + 2 * PT_KEYS * (HD + 4) + 2 * PT_KEYS * HD + 16 * RPT * (PT_KEYS + 8)) * 4; }

template <int HD, int RPT>
__global__ void __launch_bounds__(PT_THREADS, 2) attention_prompt_kernel(const PromptArgs p) {
    constexpr int PT_ROWS = 16 * RPT;
    constexpr int LQ = HD + 4, LS = PT_KEYS + 8, CH = HD / 32;         // CH: groups of four channels per thread
    extern __shared__ __align__(16) float pt[];
    float* sq = pt;                                                    // [PT_ROWS][LQ]
    float* sk = sq + PT_ROWS * LQ;                                     // [2][32][LQ]
    float* sv = sk + 2 * PT_KEYS * LQ;                                 // [2][32][HD]
    float* sp = sv + 2 * PT_KEYS * HD;                                 // [PT_ROWS][LS]
    const int seq = blockIdx.z, kvh = blockIdx.y, group = p.nq / p.nkv, tokens = PT_ROWS / group;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = lane >> 3, tx = lane & 7;
    const int r0 = p.seq_start[seq], n = p.seq_qlen[seq], pos0 = p.seq_pos0[seq];
    // the last tiles see the most keys: they start first
    const int t0 = ((n + tokens - 1) / tokens - 1 - (int)blockIdx.x) * tokens;
    fr_pdl_wait();
    fr_pdl_launch();
    if (t0 < 0 || n <= 0) return;
    const int rows = min(tokens, n - t0) * group;
    const bool ended = p.row_seq[r0] < 0;
    const int last = pos0 + t0 + rows / group - 1, lo = p.window > 0 ? max(0, pos0 + t0 - p.window + 1) : 0;
    const int steps = ended ? 0 : (last - lo) / PT_KEYS + 1;
    const int* table = p.block_table + (size_t)seq * p.table_width;
    auto copy = [&](float* dst, const float* src, bool there) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(there ? src : p.k_pool), "r"(there ? 16 : 0)
                     : "memory");
    };
    auto fetch = [&](int step) {
        float* dk = sk + (step & 1) * PT_KEYS * LQ;
        float* dv = sv + (step & 1) * PT_KEYS * HD;
        for (int idx = tid; idx < PT_KEYS * (HD / 4); idx += PT_THREADS) {
            const int key = idx / (HD / 4), c = idx % (HD / 4) * 4, j = lo + step * PT_KEYS + key;
            const bool there = j <= last && c < p.hd;
            const int jj = min(j, last);
            const size_t at = (((size_t)table[jj / p.page] * p.page + jj % p.page) * p.nkv + kvh) * p.hd + c;
            copy(dk + key * LQ + c, p.k_pool + (there ? at : 0), there);
            copy(dv + key * HD + c, p.v_pool + (there ? at : 0), there);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (steps > 0) fetch(0);
    for (int idx = tid; idx < PT_ROWS * (HD / 4); idx += PT_THREADS) {
        const int r = idx / (HD / 4), c = idx % (HD / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows && c < p.hd) v = *(const float4*)(p.q + (size_t)(r0 + t0 + r / group) * p.q_stride + (size_t)(kvh * group + r % group) * p.hd + c);
        v.x *= p.scale; v.y *= p.scale; v.z *= p.scale; v.w *= p.scale;
        *(float4*)(sq + r * LQ + c) = v;
    }
    // this thread's rows: row0 + 4 i (in shared memory four rows of a warp then lie in different banks)
    const int row0 = warp * 4 * RPT + ty;
    int pos[RPT];
    float m[RPT], l[RPT], acc[RPT][4 * CH];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        pos[i] = pos0 + t0 + min(row0 + 4 * i, rows - 1) / group;
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * CH; ++c) acc[i][c] = 0.f;
    }
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                               // this block of keys is here, and everyone is done with the one before
        if (step + 1 < steps) fetch(step + 1);
        const float* kb = sk + (step & 1) * PT_KEYS * LQ;
        const float* vb = sv + (step & 1) * PT_KEYS * HD;
        const int j0 = lo + step * PT_KEYS;
        float s[RPT][4];                                               // keys j0 + tx + 8 u
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) s[i][u] = 0.f;
#pragma unroll 1
        for (int d0 = 0; d0 < HD; d0 += 16) {
            float part[RPT][4];
#pragma unroll
            for (int d = d0; d < d0 + 16; d += 4) {
                float4 a[RPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i) a[i] = *(const float4*)(sq + (row0 + 4 * i) * LQ + d);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 b = *(const float4*)(kb + (tx + 8 * u) * LQ + d);
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        const float first = d == d0 ? a[i].w * b.w : fmaf(a[i].w, b.w, part[i][u]);
                        part[i][u] = fmaf(a[i].x, b.x, fmaf(a[i].y, b.y, fmaf(a[i].z, b.z, first)));
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int u = 0; u < 4; ++u) s[i][u] += part[i][u];
        }
        // keys that some row of the tile does not see
        const bool masked = j0 + PT_KEYS - 1 > pos0 + t0 || (p.window > 0 && j0 <= last - p.window);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (masked)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + tx + 8 * u;
                    if (j > pos[i] || (p.window > 0 && j <= pos[i] - p.window)) s[i][u] = -INFINITY;
                }
            float top = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m[i], top), base = m_new == -INFINITY ? 0.f : m_new;      // (no key seen yet)
            const float alpha = expf(m[i] - base);
            float sum = 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float e = expf(s[i][u] - base);
                sum += e;
                sp[(row0 + 4 * i) * LS + tx + 8 * u] = e;
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * CH; ++c) acc[i][c] *= alpha;
        }
        __syncwarp();                                                  // a row's weights are its own warp's
        auto add = [&](auto hidden) {
#pragma unroll 2
            for (int key = 0; key < PT_KEYS; key += 4) {
                float4 w[RPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i) w[i] = *(const float4*)(sp + (row0 + 4 * i) * LS + key);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
#pragma unroll
                    for (int g = 0; g < CH; ++g) {
                        const float4 v = *(const float4*)(vb + (key + u) * HD + 4 * tx + 32 * g);
#pragma unroll
                        for (int i = 0; i < RPT; ++i) {
                            const float e = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
                            // (a key that the row does not see adds nothing, whatever its value is)
                            if (decltype(hidden)::value == 0 || e != 0.f) {
                                acc[i][4 * g] = fmaf(e, v.x, acc[i][4 * g]);
                                acc[i][4 * g + 1] = fmaf(e, v.y, acc[i][4 * g + 1]);
                                acc[i][4 * g + 2] = fmaf(e, v.z, acc[i][4 * g + 2]);
                                acc[i][4 * g + 3] = fmaf(e, v.w, acc[i][4 * g + 3]);
                            }
                        }
                    }
                }
            }
        };
        if (masked) add(Number<1>{});
        else add(Number<0>{});
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = row0 + 4 * i;
        if (r >= rows) continue;
        const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
        float* o = p.out + ((size_t)(r0 + t0 + r / group) * p.nq + kvh * group + r % group) * p.hd;
#pragma unroll
        for (int g = 0; g < CH; ++g) {
            const int c = 4 * tx + 32 * g;
            if (c < p.hd) *(float4*)(o + c) = make_float4(acc[i][4 * g] * inv, acc[i][4 * g + 1] * inv, acc[i][4 * g + 2] * inv, acc[i][4 * g + 3] * inv);
        }
    }
}

template <int HD, int RPT>
int launch_prompt_tiles(const PromptArgs& p, int n_seqs, int max_q_len, cudaStream_t stream) {
    static std::atomic<unsigned long long> configured{0};     // devices (as bits) on which the limit has been raised
    int device = 0;
    FR_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= 64) FR_REFUSE("attention: device %d is outside the table of 64", device);
    if (!(configured.load(std::memory_order_acquire) & (1ull << device))) {
        FR_CUDA(cudaFuncSetAttribute(attention_prompt_kernel<HD, RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, prompt_smem<HD, RPT>()));
        configured.fetch_or(1ull << device, std::memory_order_release);
    }
    const int tokens = 16 * RPT / (p.nq / p.nkv);
    FR_CUDA(fr_launch(attention_prompt_kernel<HD, RPT>, dim3((max_q_len + tokens - 1) / tokens, p.nkv, n_seqs), dim3(PT_THREADS), prompt_smem<HD, RPT>(), stream, p));
    FR_CHECK_LAUNCH("attention (prompts)");
    return FR_OK;
}

// Tiles of 64 rows would leave SMs with fewer than two blocks: 32 rows, where the query heads of a kv head fit them.
bool prompt_tiles_are_few(int group, long long tiles, int sms) { return group <= 32 && tiles < 4ll * sms; }

template <int HD>
int launch_prompt(const PromptArgs& p, int n_seqs, int max_q_len, cudaStream_t stream) {
    const int sms = fr_sm_count() > 0 ? fr_sm_count() : 148, group = p.nq / p.nkv, tokens = PT_MOST_ROWS / group;
    const long long tiles = (long long)((max_q_len + tokens - 1) / tokens) * p.nkv * n_seqs;
    if (prompt_tiles_are_few(group, tiles, sms)) return launch_prompt_tiles<HD, 2>(p, n_seqs, max_q_len, stream);
    return launch_prompt_tiles<HD, 4>(p, n_seqs, max_q_len, stream);
}

template <typename T>
cudaError_t launch_attention(const AttnArgs& p, dim3 grid, cudaStream_t stream) {
    const int size = p.hd > p.vd ? p.hd : p.vd;
    void (*kernel)(AttnArgs) = size <= 32 ? attention_kernel<T, 1, 8> : size <= 64 ? attention_kernel<T, 2, 16>
                             : size <= 128 ? attention_kernel<T, 4, 8> : attention_kernel<T, 8, 4>;
    // Blocks that start while the predecessor still runs go to whichever SMs are free first.  A few blocks per SM then lie
    // unevenly for the whole call (64 rows x 28 heads of 192, 700 keys: 355 us, 274 after the predecessor's end), so only a call
    // of at most two per SM starts early.
    const int sms = fr_sm_count() > 0 ? fr_sm_count() : 148;
    if ((long long)grid.x * grid.y <= 2ll * sms) return fr_launch(kernel, grid, dim3(128), 0, stream, p);
    kernel<<<grid, 128, 0, stream>>>(p);
    return cudaGetLastError();
}

}  // namespace

// Scratch floats needed for `splits` > 1 (vd: the size of a value head).
FR_EXPORT long long attention_simt_scratch_floats(int rows, int nq, int vd, int splits) {
    return splits > 1 ? (long long)rows * nq * splits * (vd + 2) : 0;
}

// vd: size of a value head (the result is [rows][nq * vd]); keep_first: keys below it stay visible behind a window;
// out_scale multiplies the result.
FR_EXPORT int attention_simt_masked(const void* q, int q_stride, void* out, const void* k_pool, const void* v_pool,
                                    const int* block_table, int table_width, int page, const int* row_seq,
                                    const int* row_pos, int rows, int nq, int nkv, int hd, int vd, int window, int keep_first,
                                    float scale, float out_scale, int splits, float* scratch, int dtype, cudaStream_t stream) {
    if (rows <= 0) return FR_OK;
    if (hd <= 0 || hd > 32 * MOST_PER_LANE) FR_REFUSE("attention: head size %d is outside 1..%d", hd, 32 * MOST_PER_LANE);
    if (vd <= 0 || vd > 32 * MOST_PER_LANE) FR_REFUSE("attention: value size %d is outside 1..%d", vd, 32 * MOST_PER_LANE);
    if (nkv <= 0 || nq % nkv != 0) FR_REFUSE("attention: %d heads cannot share %d key/value heads", nq, nkv);
    if (splits < 1 || splits > 65535) FR_REFUSE("attention: %d splits", splits);
    if (splits > 1 && scratch == nullptr) FR_REFUSE("attention: splits need a scratch buffer");
    if (keep_first < 0) FR_REFUSE("attention: keep_first = %d", keep_first);
    AttnArgs p{q, out, k_pool, v_pool, block_table, row_seq, row_pos, scratch, table_width, page, rows, nq, nkv, hd,
               q_stride, window, splits, scale, vd, window > 0 ? keep_first : 0, out_scale};
    const int items = rows * nq;
    MergeArgs mp{scratch, out, rows, nq, vd, splits, out_scale};
    dim3 grid((items + 3) / 4, splits);
    if (dtype == FR_F32) {
        FR_CUDA(launch_attention<float>(p, grid, stream));
        FR_CHECK_LAUNCH("attention");
        if (splits > 1) FR_CUDA(fr_launch(attention_merge_kernel<float>, dim3((items + 3) / 4), dim3(128), 0, stream, mp));
    } else if (dtype == FR_BF16) {
        FR_CUDA(launch_attention<__nv_bfloat16>(p, grid, stream));
        FR_CHECK_LAUNCH("attention");
        if (splits > 1) FR_CUDA(fr_launch(attention_merge_kernel<__nv_bfloat16>, dim3((items + 3) / 4), dim3(128), 0, stream, mp));
    } else {
        FR_REFUSE("attention: unknown dtype %d", dtype);
    }
    FR_CHECK_LAUNCH("attention merge");
    return FR_OK;
}

FR_EXPORT int attention_simt(const void* q, int q_stride, void* out, const void* k_pool, const void* v_pool,
                             const int* block_table, int table_width, int page, const int* row_seq,
                             const int* row_pos, int rows, int nq, int nkv, int hd, int window, float scale,
                             int splits, float* scratch, int dtype, cudaStream_t stream) {
    return attention_simt_masked(q, q_stride, out, k_pool, v_pool, block_table, table_width, page, row_seq, row_pos, rows, nq,
                                 nkv, hd, hd, window, 0, scale, 1.0f, splits, scratch, dtype, stream);
}

// Whether attention_simt_prompt takes these sizes (rows in 16-byte pieces, a kv head's query heads within a tile).
FR_EXPORT int attention_simt_prompt_supports(const void* q, int q_stride, const void* out, const void* k_pool, const void* v_pool, int nq, int nkv,
                                             int hd, int n_seqs) {
    return hd > 0 && hd <= 128 && hd % 4 == 0 && nkv > 0 && nkv <= 65535 && nq % nkv == 0 && nq / nkv <= PT_MOST_ROWS && q_stride % 4 == 0 && n_seqs <= 65535 &&
           (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0;
}

// Whether attention_simt_prompt is the faster way for a step (max_kv_len: of the longest sequence, its new rows included; `splits`: of the
// keys by attention_simt).  Both times are estimated, in us, from what was measured on B200 at 16 to 333 new rows behind 0 to 8,000 keys, heads 28 on 4,
// 64 on 1, 8 and 16 of their own, 3 on 1:
//   a warp per row and head: a key costs a warp 0.15 (0.11 up to 64 channels) while few warps run, and the SMs do 6,800 (7,800) keys of a row
//   and head in a microsecond;
//   tiles: a block walks its keys whatever the number of its rows, 32 in 3.8 (2.4 and 1.55 up to 64 and 32 channels; of 64 rows 5.2, 3.3 and 2.1), and
//   never shares them with another block.
// So few rows behind many keys are the first one's, whose warps split the keys (16 rows behind 8,000 keys: 28 on 4 heads 489 and 945, 8 heads 155 and
// 939; 64 rows 2,414 and 947, 618 and 942; without keys before them 16 rows 4.5 and 8.2, 64 rows 16 and 12).  Over the 303 steps that were measured
// the tiles, where taken, were never more than 3 % behind, but for 100 rows beside 64 sequences of one (145 and 167).
FR_EXPORT int attention_simt_prompt_pays(int rows, int n_seqs, int max_q_len, int max_kv_len, int nq, int nkv, int hd, int window, int splits) {
    // (fewer new tokens than were measured stay where they are)
    if (rows <= 0 || n_seqs <= 0 || max_q_len < 16 || nkv <= 0 || nq < nkv || splits <= 0 || nq / nkv > PT_MOST_ROWS) return 0;
    const int sms = fr_sm_count() > 0 ? fr_sm_count() : 148, group = nq / nkv, size = hd > 64 ? 2 : hd > 32 ? 1 : 0;
    const double seen = window > 0 && window < max_kv_len ? window : max_kv_len;
    double keys = max_kv_len - 0.5 * max_q_len;               // of a row, about
    if (window > 0 && window < keys) keys = window;
    const double in_turn = (size == 2 ? 0.15 : 0.11) * ceil(seen / splits), all = (double)rows * keys * nq / (size == 2 ? 6800.0 : 7800.0);
    const double some = splits > 1 ? all : all + (in_turn < 12.0 ? 0.5 * in_turn : 6.0);        // (the rows that see little end early)
    const double by_row = (in_turn > some ? in_turn : some) + (splits > 1 ? 8.0 : 3.0);

    const long long tiles = (long long)((max_q_len + PT_MOST_ROWS / group - 1) / (PT_MOST_ROWS / group)) * nkv * n_seqs;
    const bool few = prompt_tiles_are_few(group, tiles, sms);
    const double step[2][3] = {{2.1, 3.3, 5.2}, {1.55, 2.4, 3.8}};
    const int tokens = (few ? 32 : 64) / group;
    long long blocks = (long long)((max_q_len + tokens - 1) / tokens) * n_seqs;
    if (rows / tokens + n_seqs < blocks) blocks = rows / tokens + n_seqs;
    blocks *= nkv;
    double reach = max_kv_len;
    if (window > 0 && window + tokens < reach) reach = window + tokens;
    const double tiled = (few ? 4.4 : 8.0) + ceil(reach / PT_KEYS) * step[few][size] * (double)((blocks + sms - 1) / sms);
    return tiled <= 0.95 * by_row;
}

// attention_simt for prompts in fp32: sequence s brings the rows seq_start[s] .. + seq_qlen[s] - 1 at positions from seq_pos0[s] on;
// row_seq[seq_start[s]] < 0: it has ended (its rows become zeros).
FR_EXPORT int attention_simt_prompt(const float* q, int q_stride, float* out, const float* k_pool, const float* v_pool, const int* block_table,
                                    int table_width, int page, const int* row_seq, const int* seq_start, const int* seq_qlen, const int* seq_pos0,
                                    int n_seqs, int max_q_len, int nq, int nkv, int hd, int window, float scale, cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0) return FR_OK;
    if (!attention_simt_prompt_supports(q, q_stride, out, k_pool, v_pool, nq, nkv, hd, n_seqs))
        FR_REFUSE("attention (prompts): %d heads on %d of %d, stride %d", nq, nkv, hd, q_stride);
    const PromptArgs p{q, out, k_pool, v_pool, block_table, row_seq, seq_start, seq_qlen, seq_pos0, table_width, page, nq, nkv, hd, q_stride, window, scale};
    if (hd <= 32) return launch_prompt<32>(p, n_seqs, max_q_len, stream);
    if (hd <= 64) return launch_prompt<64>(p, n_seqs, max_q_len, stream);
    return launch_prompt<128>(p, n_seqs, max_q_len, stream);
}
