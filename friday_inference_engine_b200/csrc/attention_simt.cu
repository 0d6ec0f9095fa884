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
