// Attention whose keys and values are expanded from one small latent per token.
//
// Every token leaves a latent c [rank] (RMS-normed) and one rotated key part r [rot] that all heads share; head h has
// key [W_uk,h c ; r] and value W_uv,h c.  Nothing but c and r is cached.  The expansion is never materialised: with
//     qc_h = W_uk,h^T q_h(unrotated part)                       [rank]
// the score of query i and key j is (qc_h(i) . c(j) + qr_h(i) . r(j)) * scale, and the head's result is
//     W_uv,h (sum_j p_ij c(j)) ,
// so every head attends over the same rows [c ; r] of the cache (read once per key for score and value alike).
// The softmax may have a sink per head: a logit that takes part in the denominator only (no key, no value, not scaled).
//
//   rotate_pairs   interleaved rotary encoding in place: (x[2i], x[2i+1]) of the chosen dimensions of every head turn by
//                  pos * freq[i]; cos and sin are multiplied by `mult` (frequency tables that stretch long wavelengths
//                  carry such a multiplier)
//   prepare        per row of the stacked projection [q | dkv | ...]: c = rmsnorm(dkv[:rank]) * w and the rotated r go to
//                  `ckr` [rows][rank + rot] (what the cache stores), the rotated query parts go to qf [rows][heads][rank + rot]
//                  (fp32) behind the place of qc
//   head_linear    a product per head: out[row][h][n] = sum_k x[row][h][k] W_h[k][n] (weights [heads * k][n], layout 0) or
//                  sum_k x[row][h][k] W_h[n][k] (weights [heads * n][k], layout 1), optionally times sigmoid(gate[row][h])
//   attention      a block per (row, split of the keys) that stages the cached rows for all heads (bf16, up to 32 heads), else a
//                  warp per (row, head, split): online softmax in fp32 over the paged cache
//                  (c in the key pool [pages][page][rank], r in the value pool [pages][page][rot]); a merge kernel when the
//                  keys were split; the sink joins the denominator at the end
//
// Scores, weights, norms, positions and angles are fp32; the angle is fp32(pos) * freq[i], sine and cosine by sincosf.
#include <math.h>

#include "common.cuh"

FR_EXPORT const char* attention_latent_last_error() { return fr_error_text; }

typedef __nv_bfloat16 bf16;

namespace {

// ------------------------------------------------------------------ rotation
struct RotateArgs {
    void* x;                  // [rows][ld]
    const int* row_seq;       // may be null
    const int* row_pos;
    const float* freq;        // [dims / 2]
    float mult;
    int ld, rows, heads, head_stride, first, dims;
};

template <typename T>
__global__ void rotate_pairs_kernel(RotateArgs p) {
    fr_pdl_wait();
    fr_pdl_launch();
    const int row = blockIdx.x;
    if (p.row_seq != nullptr && p.row_seq[row] < 0) return;
    const float pos = (float)p.row_pos[row];
    const int half = p.dims / 2;
    T* x = (T*)p.x + (size_t)row * p.ld;
    for (int idx = threadIdx.x; idx < p.heads * half; idx += blockDim.x) {
        const int h = idx / half, i = idx - h * half;
        float s, c;
        sincosf(pos * p.freq[i], &s, &c);
        s *= p.mult;
        c *= p.mult;
        T* at = x + (size_t)h * p.head_stride + p.first + 2 * i;
        float a, b;
        fr_rotate(fr_load(at), fr_load(at + 1), c, s, a, b);
        fr_store(at, a);
        fr_store(at + 1, b);
    }
}

// ------------------------------------------------------------------ prepare
struct PrepareArgs {
    const void* x;            // [rows][ld]: queries [heads][dim + rot] at q_off, [latent rank | key part rot] at kv_off
    void* ckr;                // [rows][rank + rot] in x's dtype
    float* qf;                // [rows][heads][rank + rot] fp32: this kernel fills the last rot of every head
    const void* norm_w;       // [rank]
    int norm_dtype;
    const int* row_seq;
    const int* row_pos;
    const float* freq;        // [rot / 2]
    float mult, eps;
    int ld, q_off, kv_off, heads, dim, rot, rank;
    int rot_dims;             // the first rot_dims of the rot numbers turn, the rest pass unchanged
};

template <typename T>
__global__ void __launch_bounds__(256) prepare_kernel(PrepareArgs p) {
    __shared__ float partial[8];
    fr_pdl_wait();
    fr_pdl_launch();
    const int row = blockIdx.x;
    if (p.row_seq != nullptr && p.row_seq[row] < 0) return;
    const T* x = (const T*)p.x + (size_t)row * p.ld;
    T* ckr = (T*)p.ckr + (size_t)row * (p.rank + p.rot);
    float ss = 0.f;
    for (int i = threadIdx.x; i < p.rank; i += blockDim.x) {
        const float v = fr_load(x + p.kv_off + i);
        ss = fmaf(v, v, ss);
    }
    ss = fr_warp_sum(ss);
    if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) total += partial[i];
    const float inv = 1.0f / sqrtf(total / (float)p.rank + p.eps);
    const FrVec w{p.norm_w, p.norm_dtype};
    for (int i = threadIdx.x; i < p.rank; i += blockDim.x) fr_store(ckr + i, fr_load(x + p.kv_off + i) * inv * w.at(i));
    const float pos = (float)p.row_pos[row];
    const int half = p.rot_dims / 2;
    // what does not turn passes as it is
    const int still = p.rot - p.rot_dims;
    for (int idx = threadIdx.x; idx < (p.heads + 1) * still; idx += blockDim.x) {
        const int item = idx / still, e = p.rot_dims + (idx - item * still);
        if (item == 0) ckr[p.rank + e] = x[p.kv_off + p.rank + e];
        else p.qf[((size_t)row * p.heads + item - 1) * (p.rank + p.rot) + p.rank + e] = fr_load(x + p.q_off + (size_t)(item - 1) * (p.dim + p.rot) + p.dim + e);
    }
    // the key part (item 0) and every head's rotated query part
    for (int idx = threadIdx.x; idx < (p.heads + 1) * half; idx += blockDim.x) {
        const int item = idx / half, i = idx - item * half;
        float s, c;
        sincosf(pos * p.freq[i], &s, &c);
        s *= p.mult;
        c *= p.mult;
        float a, b;
        if (item == 0) {
            fr_rotate(fr_load(x + p.kv_off + p.rank + 2 * i), fr_load(x + p.kv_off + p.rank + 2 * i + 1), c, s, a, b);
            fr_store(ckr + p.rank + 2 * i, a);
            fr_store(ckr + p.rank + 2 * i + 1, b);
        } else {
            const int h = item - 1;
            const T* q = x + p.q_off + (size_t)h * (p.dim + p.rot) + p.dim + 2 * i;
            fr_rotate(fr_load(q), fr_load(q + 1), c, s, a, b);
            float* o = p.qf + ((size_t)row * p.heads + h) * (p.rank + p.rot) + p.rank + 2 * i;
            o[0] = a;
            o[1] = b;
        }
    }
}

// ------------------------------------------------------------------ a product per head
struct HeadLinearArgs {
    const void* x;            // [rows][ld_x], head h at x_off + h * x_stride, k numbers
    const void* w;            // layout 0: [heads * k][n]; layout 1: [heads * n][k]
    void* out;                // [rows][ld_out], head h at h * out_stride, n numbers
    const void* gate;         // [rows][ld_gate] at gate_off + h: the result is multiplied by its sigmoid (or null)
    const int* row_seq;
    int rows, heads, k, n, ld_x, x_off, x_stride, ld_out, out_stride, ld_gate, gate_off;
    int fixed_weights;        // no kernel writes w any more: it may be read ahead of the wait for the kernel before
};

constexpr int HL_ROWS = 8;        // rows per block

// layout 0: a thread owns output column n of head blockIdx.y for HL_ROWS rows; x staged in shared memory
template <typename TX, typename TW, typename TO, typename TG>
__global__ void __launch_bounds__(128) head_linear_kn_kernel(HeadLinearArgs p) {
    extern __shared__ float sx[];            // [HL_ROWS][k]
    fr_pdl_wait();
    fr_pdl_launch();
    const int h = blockIdx.y, row0 = blockIdx.z * HL_ROWS;
    const int nr = min(HL_ROWS, p.rows - row0);
    for (int idx = threadIdx.x; idx < nr * p.k; idx += blockDim.x) {
        const int r = idx / p.k, i = idx - r * p.k;
        sx[r * p.k + i] = fr_load((const TX*)p.x + (size_t)(row0 + r) * p.ld_x + p.x_off + (size_t)h * p.x_stride + i);
    }
    __syncthreads();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= p.n) return;
    float acc[HL_ROWS];
#pragma unroll
    for (int r = 0; r < HL_ROWS; ++r) acc[r] = 0.f;
    const TW* w = (const TW*)p.w + (size_t)h * p.k * p.n + n;
    for (int i = 0; i < p.k; ++i) {
        const float wv = fr_load(w + (size_t)i * p.n);
#pragma unroll
        for (int r = 0; r < HL_ROWS; ++r)
            if (r < nr) acc[r] = fmaf(sx[r * p.k + i], wv, acc[r]);
    }
#pragma unroll
    for (int r = 0; r < HL_ROWS; ++r) {
        if (r >= nr) continue;
        const int row = row0 + r;
        if (p.row_seq != nullptr && p.row_seq[row] < 0) continue;
        float v = acc[r];
        if (p.gate != nullptr) {
            const float g = fr_load((const TG*)p.gate + (size_t)row * p.ld_gate + p.gate_off + h);
            v *= 1.0f / (1.0f + expf(-g));
        }
        fr_store((TO*)p.out + (size_t)row * p.ld_out + (size_t)h * p.out_stride + n, v);
    }
}

// layout 1: a warp owns output column n of head blockIdx.y for HL_ROWS rows; the lanes share k
template <typename TX, typename TW, typename TO, typename TG>
__global__ void __launch_bounds__(128) head_linear_nk_kernel(HeadLinearArgs p) {
    extern __shared__ float sx[];            // [HL_ROWS][k]
    fr_pdl_wait();
    fr_pdl_launch();
    const int h = blockIdx.y, row0 = blockIdx.z * HL_ROWS;
    const int nr = min(HL_ROWS, p.rows - row0);
    for (int idx = threadIdx.x; idx < nr * p.k; idx += blockDim.x) {
        const int r = idx / p.k, i = idx - r * p.k;
        sx[r * p.k + i] = fr_load((const TX*)p.x + (size_t)(row0 + r) * p.ld_x + p.x_off + (size_t)h * p.x_stride + i);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int n = blockIdx.x * 16 + warp; n < min(p.n, (int)(blockIdx.x + 1) * 16); n += 4) {
        float acc[HL_ROWS];
#pragma unroll
        for (int r = 0; r < HL_ROWS; ++r) acc[r] = 0.f;
        const TW* w = (const TW*)p.w + ((size_t)h * p.n + n) * p.k;
        for (int i = lane; i < p.k; i += 32) {
            const float wv = fr_load(w + i);
#pragma unroll
            for (int r = 0; r < HL_ROWS; ++r)
                if (r < nr) acc[r] = fmaf(sx[r * p.k + i], wv, acc[r]);
        }
#pragma unroll
        for (int r = 0; r < HL_ROWS; ++r) acc[r] = fr_warp_sum(acc[r]);
        if (lane == 0) {
#pragma unroll
            for (int r = 0; r < HL_ROWS; ++r) {
                if (r >= nr) continue;
                const int row = row0 + r;
                if (p.row_seq != nullptr && p.row_seq[row] < 0) continue;
                float v = acc[r];
                if (p.gate != nullptr) {
                    const float g = fr_load((const TG*)p.gate + (size_t)row * p.ld_gate + p.gate_off + h);
                    v *= 1.0f / (1.0f + expf(-g));
                }
                fr_store((TO*)p.out + (size_t)row * p.ld_out + (size_t)h * p.out_stride + n, v);
            }
        }
    }
}

// The same two products for bf16 weights in 16-byte pieces, with the weights of a thread (fixed ones) on their way before the
// predecessor has finished: a decoding step runs one round of blocks, so the chain of waits is the cost (8 rows, 16 heads, 128 x 512: 22 us each
// with the kernels above, 5.8 and 8.8 with these).
__device__ __forceinline__ void eight_of(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <typename TX>
__device__ __forceinline__ void stage_rows(const HeadLinearArgs& p, int h, int row0, int nr, float* sx) {
    for (int idx = threadIdx.x; idx < HL_ROWS * p.k; idx += blockDim.x) {
        const int r = idx / p.k, i = idx - r * p.k;
        sx[idx] = r < nr ? fr_load((const TX*)p.x + (size_t)(row0 + r) * p.ld_x + p.x_off + (size_t)h * p.x_stride + i) : 0.f;
    }
}
template <typename TO>
__device__ __forceinline__ void head_out(const HeadLinearArgs& p, int row, int h, int n, float v) {
    if (p.row_seq != nullptr && p.row_seq[row] < 0) return;
    if (p.gate != nullptr) {
        const float g = fr_load((const TO*)p.gate + (size_t)row * p.ld_gate + p.gate_off + h);
        v *= 1.0f / (1.0f + expf(-g));
    }
    fr_store((TO*)p.out + (size_t)row * p.ld_out + (size_t)h * p.out_stride + n, v);
}

// layout 0: 128 columns per block, eight per thread; sixteen groups of threads share k
template <typename TX, typename TO>
__global__ void __launch_bounds__(256) head_kn_kernel(HeadLinearArgs p) {
    extern __shared__ __align__(16) float sx[];          // [HL_ROWS][k], then [8 warps][HL_ROWS][128]
    float* red = sx + HL_ROWS * p.k;
    const int h = blockIdx.y, row0 = blockIdx.z * HL_ROWS, nr = min(HL_ROWS, p.rows - row0);
    const int group = threadIdx.x >> 4, c0 = (threadIdx.x & 15) * 8, n0 = blockIdx.x * 128;
    const bool inside = n0 + c0 < p.n;
    const bf16* w = (const bf16*)p.w + (size_t)h * p.k * p.n + (inside ? n0 + c0 : 0);
    uint4 wv[8];
    auto fetch = [&](int i0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + group + 16 * u;
            wv[u] = i < p.k ? __ldg((const uint4*)(w + (size_t)i * p.n)) : make_uint4(0, 0, 0, 0);
        }
    };
    if (!p.fixed_weights) fr_pdl_wait();
    fetch(0);
    fr_pdl_wait();
    fr_pdl_launch();
    stage_rows<TX>(p, h, row0, nr, sx);
    __syncthreads();
    float acc[HL_ROWS][8];
#pragma unroll
    for (int r = 0; r < HL_ROWS; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[r][e] = 0.f;
    for (int i0 = 0; i0 < p.k; i0 += 128) {
        if (i0 > 0) fetch(i0);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + group + 16 * u;
            if (i >= p.k) break;
            float f[8];
            eight_of(wv[u], f);
#pragma unroll
            for (int r = 0; r < HL_ROWS; ++r) {
                const float x = sx[r * p.k + i];
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[r][e] = fmaf(x, f[e], acc[r][e]);
            }
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < HL_ROWS; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = acc[r][e] + __shfl_xor_sync(0xffffffffu, acc[r][e], 16);
            if (lane < 16) red[(warp * HL_ROWS + r) * 128 + c0 + e] = v;
        }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nr * 128; idx += 256) {
        const int r = idx >> 7, c = idx & 127;
        if (n0 + c >= p.n) continue;
        float v = 0.f;
#pragma unroll
        for (int g = 0; g < 8; ++g) v += red[(g * HL_ROWS + r) * 128 + c];
        head_out<TO>(p, row0 + r, h, n0 + c, v);
    }
}

// layout 1: sixteen columns per block, two per warp; the lanes share k
template <typename TX, typename TO>
__global__ void __launch_bounds__(256) head_nk_kernel(HeadLinearArgs p) {
    extern __shared__ __align__(16) float sx[];          // [HL_ROWS][k]
    const int h = blockIdx.y, row0 = blockIdx.z * HL_ROWS, nr = min(HL_ROWS, p.rows - row0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = blockIdx.x * 16 + 2 * warp;
    const uint4* w[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) w[c] = (const uint4*)((const bf16*)p.w + ((size_t)h * p.n + min(n0 + c, p.n - 1)) * p.k);
    const int pieces = p.k >> 3;
    uint4 wv[2][2];
    auto fetch = [&](int q0) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int u = 0; u < 2; ++u) wv[c][u] = q0 + lane + 32 * u < pieces ? __ldg(w[c] + q0 + lane + 32 * u) : make_uint4(0, 0, 0, 0);
    };
    if (!p.fixed_weights) fr_pdl_wait();
    fetch(0);
    fr_pdl_wait();
    fr_pdl_launch();
    stage_rows<TX>(p, h, row0, nr, sx);
    __syncthreads();
    float acc[2 * HL_ROWS];                              // [row][column]
#pragma unroll
    for (int v = 0; v < 2 * HL_ROWS; ++v) acc[v] = 0.f;
    for (int q0 = 0; q0 < pieces; q0 += 64) {
        if (q0 > 0) fetch(q0);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + lane + 32 * u;
            if (q >= pieces) break;
            float f[2][8];
            eight_of(wv[0][u], f[0]);
            eight_of(wv[1][u], f[1]);
#pragma unroll
            for (int r = 0; r < HL_ROWS; ++r) {
                const float4 a = *(const float4*)(sx + r * p.k + 8 * q), b = *(const float4*)(sx + r * p.k + 8 * q + 4);
                const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[2 * r + c] = fmaf(x[e], f[c][e], acc[2 * r + c]);
            }
        }
    }
    // sums over the lanes: halve the values and double the lanes behind each; lanes 2 v and 2 v + 1 end with value v
#pragma unroll
    for (int half = HL_ROWS, bit = 16; half > 0; half >>= 1, bit >>= 1)
#pragma unroll
        for (int v = 0; v < HL_ROWS; ++v)
            if (v < half) {
                const bool upper = (lane & bit) != 0;
                const float give = upper ? acc[v] : acc[v + half], keep = upper ? acc[v + half] : acc[v];
                acc[v] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
            }
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
    const int value = lane >> 1, r = value >> 1, n = n0 + (value & 1);
    if ((lane & 1) == 0 && r < nr && n < p.n) head_out<TO>(p, row0 + r, h, n, acc[0]);
}

template <typename TX, typename TO>
int launch_head_pieces(const HeadLinearArgs& p, int layout, cudaStream_t stream) {
    const int row_blocks = (p.rows + HL_ROWS - 1) / HL_ROWS;
    const size_t rows = (size_t)HL_ROWS * p.k * sizeof(float);
    if (layout == 0) {
        const size_t smem = rows + 8 * HL_ROWS * 128 * sizeof(float);
        if (smem > 48 * 1024) FR_CUDA(cudaFuncSetAttribute(head_kn_kernel<TX, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        FR_CUDA(fr_launch(head_kn_kernel<TX, TO>, dim3((p.n + 127) / 128, p.heads, row_blocks), dim3(256), smem, stream, p));
    } else {
        FR_CUDA(fr_launch(head_nk_kernel<TX, TO>, dim3((p.n + 15) / 16, p.heads, row_blocks), dim3(256), rows, stream, p));
    }
    FR_CHECK_LAUNCH("head_linear (pieces)");
    return FR_OK;
}

template <typename TX, typename TW, typename TO>
int launch_head_linear(const HeadLinearArgs& p, int layout, cudaStream_t stream) {
    const size_t smem = (size_t)HL_ROWS * p.k * sizeof(float);
    if (smem > 48 * 1024) FR_REFUSE("head_linear: %d inputs per head (at most %d)", p.k, 48 * 1024 / (HL_ROWS * 4));
    const int row_blocks = (p.rows + HL_ROWS - 1) / HL_ROWS;
    if (layout == 0) {
        const dim3 grid((p.n + 127) / 128, p.heads, row_blocks);
        FR_CUDA(fr_launch(head_linear_kn_kernel<TX, TW, TO, TO>, grid, dim3(128), smem, stream, p));
    } else {
        const dim3 grid((p.n + 15) / 16, p.heads, row_blocks);
        FR_CUDA(fr_launch(head_linear_nk_kernel<TX, TW, TO, TO>, grid, dim3(128), smem, stream, p));
    }
    FR_CHECK_LAUNCH("head_linear");
    return FR_OK;
}

// ------------------------------------------------------------------ attention
constexpr int C_PER_LANE = 16;    // latent sizes up to 512
constexpr int R_PER_LANE = 4;     // rotated key parts up to 128

struct AttnArgs {
    const float* q;           // [rows][heads][rank + rot]
    float* out;               // [rows][heads][rank]
    const void* c_pool;       // [pages][page][rank]
    const void* r_pool;       // [pages][page][rot]
    const int* block_table;
    const int* row_seq;
    const int* row_pos;
    const void* sink;         // [heads] or null
    int sink_dtype;
    float* part;              // [rows * heads][splits][rank + 2] when splits > 1
    int table_width, page, rows, heads, rank, rot, splits;
    float scale;
};

// V numbers per lane and load: lane l owns dimensions V l + e + 32 V i (e < V).  V = 2 needs an even latent size and an
// even rotated part (rows of the pools then start on 4-byte boundaries).
template <typename T, int V> struct Pack;
template <> struct Pack<float, 1> { static __device__ __forceinline__ void load(const float* p, float* o) { o[0] = *p; } };
template <> struct Pack<bf16, 1> { static __device__ __forceinline__ void load(const bf16* p, float* o) { o[0] = __bfloat162float(*p); } };
template <> struct Pack<float, 2> {
    static __device__ __forceinline__ void load(const float* p, float* o) { const float2 v = *(const float2*)p; o[0] = v.x; o[1] = v.y; }
};
template <> struct Pack<bf16, 2> {
    static __device__ __forceinline__ void load(const bf16* p, float* o) {
        const float2 v = __bfloat1622float2(*(const __nv_bfloat162*)p);
        o[0] = v.x; o[1] = v.y;
    }
};

template <typename T, int V>
__global__ void __launch_bounds__(128) latent_attention_kernel(AttnArgs p) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * 4 + warp;          // (row, head)
    if (item >= p.rows * p.heads) return;
    const int row = item / p.heads, h = item - row * p.heads;
    const int split = blockIdx.y;
    fr_pdl_wait();
    fr_pdl_launch();
    const int seq = p.row_seq[row];
    constexpr int CI = C_PER_LANE / V, RI = R_PER_LANE / V;
    float qc[C_PER_LANE], qr[R_PER_LANE], acc[C_PER_LANE];
#pragma unroll
    for (int i = 0; i < C_PER_LANE; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;
    if (seq >= 0) {
        const int n = p.row_pos[row] + 1;
        const int chunk = (n + p.splits - 1) / p.splits;
        const int i0 = split * chunk, i1 = min(i0 + chunk, n);
        const float* q = p.q + (size_t)item * (p.rank + p.rot);
#pragma unroll
        for (int i = 0; i < CI; ++i)
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int d = V * lane + 32 * V * i + e;
                qc[V * i + e] = d < p.rank ? q[d] * p.scale : 0.f;
            }
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int d = V * lane + 32 * V * i + e;
                qr[V * i + e] = d < p.rot ? q[p.rank + d] * p.scale : 0.f;
            }
        const int* table = p.block_table + (size_t)seq * p.table_width;
        // two keys at a time: their loads are issued together
        for (int j = i0; j < i1; j += 2) {
            float cv[2][C_PER_LANE], s2[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int ju = min(j + u, i1 - 1);
                const size_t at = (size_t)table[ju / p.page] * p.page + ju % p.page;
                const T* cr = (const T*)p.c_pool + at * p.rank;
                const T* rr = (const T*)p.r_pool + at * p.rot;
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < CI; ++i) {
                    const int d = V * lane + 32 * V * i;
#pragma unroll
                    for (int e = 0; e < V; ++e) cv[u][V * i + e] = 0.f;
                    if (d < p.rank) Pack<T, V>::load(cr + d, &cv[u][V * i]);
#pragma unroll
                    for (int e = 0; e < V; ++e) s = fmaf(qc[V * i + e], cv[u][V * i + e], s);
                }
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const int d = V * lane + 32 * V * i;
                    float rv[V];
#pragma unroll
                    for (int e = 0; e < V; ++e) rv[e] = 0.f;
                    if (d < p.rot) Pack<T, V>::load(rr + d, rv);
#pragma unroll
                    for (int e = 0; e < V; ++e) s = fmaf(qr[V * i + e], rv[e], s);
                }
                s2[u] = s;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s2[0] += __shfl_xor_sync(0xffffffffu, s2[0], o);
                s2[1] += __shfl_xor_sync(0xffffffffu, s2[1], o);
            }
            const bool two = j + 1 < i1;
            const float m_new = fmaxf(m, two ? fmaxf(s2[0], s2[1]) : s2[0]);
            const float alpha = expf(m - m_new);
            const float e0 = expf(s2[0] - m_new), e1 = two ? expf(s2[1] - m_new) : 0.f;
            l = l * alpha + (e0 + e1);
#pragma unroll
            for (int i = 0; i < C_PER_LANE; ++i) acc[i] = acc[i] * alpha + (e0 * cv[0][i] + e1 * cv[1][i]);
            m = m_new;
        }
    }
    if (p.splits > 1) {
        float* part = p.part + ((size_t)item * p.splits + split) * (p.rank + 2);
#pragma unroll
        for (int i = 0; i < CI; ++i)
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const int d = V * lane + 32 * V * i + e;
                if (d < p.rank) part[d] = acc[V * i + e];
            }
        if (lane == 0) {
            part[p.rank] = m;
            part[p.rank + 1] = l;
        }
        return;
    }
    float* o = p.out + (size_t)item * p.rank;
    float denom = l;
    float f = 1.f;
    if (p.sink != nullptr && seq >= 0) {
        const float sk = FrVec{p.sink, p.sink_dtype}.at(h);
        const float top = fmaxf(m, sk);
        f = expf(m - top);
        denom = l * f + expf(sk - top);
    }
    const float inv = denom > 0.f ? f / denom : 0.f;
#pragma unroll
    for (int i = 0; i < CI; ++i)
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const int d = V * lane + 32 * V * i + e;
            if (d < p.rank) o[d] = acc[V * i + e] * inv;
        }
}

// The same for a bf16 cache, all heads of a row in one block: the block brings KEYS cached rows at a time into shared memory (the
// next ones on their way meanwhile), and its warps take the heads in turn, NH each.  A warp per (row, head) read every cached
// row once per head, two at a time: 8 rows, 16 heads, up to 540 keys took 47 us, 20 here.
constexpr int KEYS = 16;
template <int NH>
__global__ void __launch_bounds__(256, NH <= 2 ? 2 : 1) latent_rows_kernel(AttnArgs p) {
    extern __shared__ __align__(16) unsigned char keys_raw[];            // [2][KEYS][rank + rot] bf16
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x, split = blockIdx.y;
    const int width = p.rank + p.rot;
    bf16* keys = (bf16*)keys_raw;
    fr_pdl_wait();
    fr_pdl_launch();
    const int seq = p.row_seq[row];
    const int n = seq >= 0 ? p.row_pos[row] + 1 : 0, chunk = (n + p.splits - 1) / p.splits;
    const int i0 = min(split * chunk, n), i1 = min(i0 + chunk, n);
    const int* table = p.block_table + (size_t)max(seq, 0) * p.table_width;
    auto fetch = [&](int j0, int buf) {                                  // cached rows j0 .. j0 + KEYS - 1 of this split
        const int per = width >> 3;
        for (int idx = threadIdx.x; idx < KEYS * per; idx += 256) {
            const int u = idx / per, c = (idx - u * per) * 8;
            if (j0 + u >= i1) break;
            const size_t at = (size_t)table[(j0 + u) / p.page] * p.page + (j0 + u) % p.page;
            const bf16* src = c < p.rank ? (const bf16*)p.c_pool + at * p.rank + c : (const bf16*)p.r_pool + at * p.rot + (c - p.rank);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(keys + ((size_t)buf * KEYS + u) * width + c)), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(i0, 0);
    // lane l has dimensions 2 l, 2 l + 1 of every 64
    float q[NH][C_PER_LANE + R_PER_LANE], acc[NH][C_PER_LANE], m[NH], l[NH];
#pragma unroll
    for (int a = 0; a < NH; ++a) {
        const int h = warp + 8 * a;
        const float* qh = p.q + ((size_t)row * p.heads + min(h, p.heads - 1)) * width;
#pragma unroll
        for (int i = 0; i < C_PER_LANE / 2; ++i) {
            const int d = 2 * lane + 64 * i;
            q[a][2 * i] = d < p.rank ? qh[d] * p.scale : 0.f;
            q[a][2 * i + 1] = d < p.rank ? qh[d + 1] * p.scale : 0.f;
        }
#pragma unroll
        for (int i = 0; i < R_PER_LANE / 2; ++i) {
            const int d = 2 * lane + 64 * i;
            q[a][C_PER_LANE + 2 * i] = d < p.rot ? qh[p.rank + d] * p.scale : 0.f;
            q[a][C_PER_LANE + 2 * i + 1] = d < p.rot ? qh[p.rank + d + 1] * p.scale : 0.f;
        }
#pragma unroll
        for (int i = 0; i < C_PER_LANE; ++i) acc[a][i] = 0.f;
        m[a] = -INFINITY;
        l[a] = 0.f;
    }
    int buf = 0;
    for (int j0 = i0; j0 < i1; j0 += KEYS, buf ^= 1) {
        fetch(j0 + KEYS, buf ^ 1);                                       // (nothing beyond the split's end)
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const bf16* rows = keys + (size_t)buf * KEYS * width;
        const int count = min(KEYS, i1 - j0);
        // (four keys of the round at a time: unrolled over all of them the loop was longer than the instruction cache, 40 us)
#pragma unroll 1
        for (int g = 0; g < count; g += 4) {
            const bf16* group = rows + (size_t)g * width + 2 * lane;
            const int live = count - g;
#pragma unroll
            for (int a = 0; a < NH; ++a) {
                if (warp + 8 * a >= p.heads) break;
                float s[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    s[u] = 0.f;
                    const bf16* kr = group + (size_t)(u < live ? u : 0) * width;
#pragma unroll
                    for (int i = 0; i < C_PER_LANE / 2; ++i) {
                        if (2 * lane + 64 * i < p.rank) {
                            const float2 c = __bfloat1622float2(*(const __nv_bfloat162*)(kr + 64 * i));
                            s[u] = fmaf(q[a][2 * i], c.x, s[u]);
                            s[u] = fmaf(q[a][2 * i + 1], c.y, s[u]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < R_PER_LANE / 2; ++i) {
                        if (2 * lane + 64 * i < p.rot) {
                            const float2 c = __bfloat1622float2(*(const __nv_bfloat162*)(kr + p.rank + 64 * i));
                            s[u] = fmaf(q[a][C_PER_LANE + 2 * i], c.x, s[u]);
                            s[u] = fmaf(q[a][C_PER_LANE + 2 * i + 1], c.y, s[u]);
                        }
                    }
                }
                // sums over the lanes: eight lanes in a row end with one key's score
                const bool up16 = (lane & 16) != 0, up8 = (lane & 8) != 0;
                const float a0 = (up16 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, up16 ? s[0] : s[2], 16);
                const float a1 = (up16 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, up16 ? s[1] : s[3], 16);
                float mine = (up8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up8 ? a0 : a1, 8);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
                if ((lane >> 3) >= live) mine = -INFINITY;
                float m_new = fmaxf(mine, __shfl_xor_sync(0xffffffffu, mine, 16));
                m_new = fmaxf(m[a], fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 8)));
                const float e = (lane >> 3) < live ? expf(mine - m_new) : 0.f, alpha = expf(m[a] - m_new);
                float w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) w[u] = __shfl_sync(0xffffffffu, e, 8 * u);
                l[a] = l[a] * alpha + ((w[0] + w[1]) + (w[2] + w[3]));
                m[a] = m_new;
#pragma unroll
                for (int i = 0; i < C_PER_LANE / 2; ++i) {
                    if (2 * lane + 64 * i < p.rank) {
                        float x = acc[a][2 * i] * alpha, y = acc[a][2 * i + 1] * alpha;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float2 c = __bfloat1622float2(*(const __nv_bfloat162*)(group + (size_t)(u < live ? u : 0) * width + 64 * i));
                            x = fmaf(w[u], c.x, x);
                            y = fmaf(w[u], c.y, y);
                        }
                        acc[a][2 * i] = x;
                        acc[a][2 * i + 1] = y;
                    }
                }
            }
        }
        __syncthreads();                                                 // all have read what the next turn overwrites
    }
#pragma unroll
    for (int a = 0; a < NH; ++a) {
        const int h = warp + 8 * a;
        if (h >= p.heads) break;
        const size_t item = (size_t)row * p.heads + h;
        float f = 1.f;
        float* o = p.out + item * p.rank;
        if (p.splits > 1) {
            o = p.part + (item * p.splits + split) * (p.rank + 2);
            if (lane == 0) {
                o[p.rank] = m[a];
                o[p.rank + 1] = l[a];
            }
        } else {
            float denom = l[a], g = 1.f;
            if (p.sink != nullptr && seq >= 0) {
                const float sk = FrVec{p.sink, p.sink_dtype}.at(h), top = fmaxf(m[a], sk);
                g = expf(m[a] - top);
                denom = l[a] * g + expf(sk - top);
            }
            f = denom > 0.f ? g / denom : 0.f;
        }
#pragma unroll
        for (int i = 0; i < C_PER_LANE / 2; ++i) {
            const int d = 2 * lane + 64 * i;
            if (d < p.rank) {
                o[d] = acc[a][2 * i] * f;
                o[d + 1] = acc[a][2 * i + 1] * f;
            }
        }
    }
}

// A block per (row, head): the splits' factors through shared memory, then every thread's dimensions with their loads in flight
// together (a warp per item walked the splits one by one: 21 us for 128 items, 7 here).
__global__ void __launch_bounds__(256) latent_merge_kernel(AttnArgs p) {
    __shared__ float factor[256];
    fr_pdl_wait();
    fr_pdl_launch();
    const int lane = threadIdx.x & 31, item = blockIdx.x, h = item % p.heads;
    const size_t step = p.rank + 2;
    const float* part = p.part + (size_t)item * p.splits * step;
    // thread s has split s (and s + 256, ...): the maximum over the block, then the factors and the sum of the weights
    __shared__ float over[2][8];
    float m_of = -INFINITY, l_of = 0.f;
    if ((int)threadIdx.x < p.splits) {
        m_of = part[threadIdx.x * step + p.rank];
        l_of = part[threadIdx.x * step + p.rank + 1];
    }
    float top = m_of;
    for (int s = threadIdx.x + 256; s < p.splits; s += 256) top = fmaxf(top, part[s * step + p.rank]);
    const bool live = p.row_seq[item / p.heads] >= 0;
    const float sk = p.sink != nullptr && live ? FrVec{p.sink, p.sink_dtype}.at(h) : -INFINITY;
    top = fr_warp_max(top);
    if (lane == 0) over[0][threadIdx.x >> 5] = top;
    __syncthreads();
    top = sk;
#pragma unroll
    for (int i = 0; i < 8; ++i) top = fmaxf(top, over[0][i]);
    float l = l_of > 0.f ? l_of * expf(m_of - top) : 0.f;
    for (int s = threadIdx.x + 256; s < p.splits; s += 256) {
        const float ls = part[s * step + p.rank + 1];
        if (ls > 0.f) l += ls * expf(part[s * step + p.rank] - top);
    }
    l = fr_warp_sum(l);
    if (lane == 0) over[1][threadIdx.x >> 5] = l;
    static_assert(32 * C_PER_LANE <= 512, "two dimensions per thread");
    const int d0 = threadIdx.x, d1 = threadIdx.x + 256;
    float a0 = 0.f, a1 = 0.f;
    for (int s0 = 0; s0 < p.splits; s0 += 256) {
        const int s = s0 + threadIdx.x, count = min(256, p.splits - s0);
        if (s0 > 0) {
            __syncthreads();
            m_of = s < p.splits ? part[s * step + p.rank] : -INFINITY;
            l_of = s < p.splits ? part[s * step + p.rank + 1] : 0.f;
        }
        factor[threadIdx.x] = l_of > 0.f ? expf(m_of - top) : 0.f;
        __syncthreads();
        const float* ps = part + s0 * step;
#pragma unroll 16
        for (int u = 0; u < count; ++u) {
            if (d0 < p.rank) a0 = fmaf(ps[u * step + d0], factor[u], a0);
            if (d1 < p.rank) a1 = fmaf(ps[u * step + d1], factor[u], a1);
        }
    }
    l = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) l += over[1][i];
    if (p.sink != nullptr && live) l += expf(sk - top);
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    float* o = p.out + (size_t)item * p.rank;
    if (d0 < p.rank) o[d0] = a0 * inv;
    if (d1 < p.rank) o[d1] = a1 * inv;
}

// Whether latent_rows_kernel takes a cache: bf16 rows in 16-byte pieces, at most 32 heads.
inline bool shared_rows(int heads, int rank, int rot, int dtype) { return dtype == FR_BF16 && heads <= 32 && rank % 8 == 0 && rot % 8 == 0; }

template <int NH>
cudaError_t launch_rows(const AttnArgs& p, cudaStream_t stream) {
    return fr_launch(latent_rows_kernel<NH>, dim3(p.rows, p.splits), dim3(256), (size_t)2 * KEYS * (p.rank + p.rot) * 2, stream, p);
}

// ------------------------------------------------------------------ prompts: the pieces between tensor-core products
// Rows [0, n) of one sequence's cached latents and key parts, gathered from the pages into contiguous rows; rows
// [n, n_pad) are zero.  The latents are written twice, [2 n_pad][rank] with row n_pad + j equal to row j: the values
// expanded from them then stand side by side twice, once for each half of the split weights.
template <typename T>
__global__ void gather_kernel(const T* __restrict__ c_pool, const T* __restrict__ r_pool, const int* __restrict__ table, int page,
                              int n, int n_pad, int rank, int rot, T* __restrict__ c_all, T* __restrict__ r_all) {
    fr_pdl_wait();
    fr_pdl_launch();
    const int j = blockIdx.x;
    T* c = c_all + (size_t)j * rank;
    T* c2 = c_all + (size_t)(n_pad + j) * rank;
    T* r = r_all + (size_t)j * rot;
    if (j >= n) {
        for (int i = threadIdx.x; i < rank; i += blockDim.x) { fr_store(c + i, 0.f); fr_store(c2 + i, 0.f); }
        for (int i = threadIdx.x; i < rot; i += blockDim.x) fr_store(r + i, 0.f);
        return;
    }
    const size_t at = (size_t)table[j / page] * page + j % page;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) { const T v = c_pool[at * rank + i]; c[i] = v; c2[i] = v; }
    for (int i = threadIdx.x; i < rot; i += blockDim.x) r[i] = r_pool[at * rot + i];
}

// Every head's key [unrotated part from kn [rows][heads * dim] | the shared rotated part r [rows][rot]] side by side:
// out [rows][heads][dim + rot]
template <typename T>
__global__ void key_concat_kernel(const T* __restrict__ kn, const T* __restrict__ r, int heads, int dim, int rot, T* __restrict__ out) {
    fr_pdl_wait();
    fr_pdl_launch();
    const size_t j = blockIdx.x;
    const int hd = dim + rot;
    for (int idx = threadIdx.x; idx < heads * hd; idx += blockDim.x) {
        const int h = idx / hd, e = idx - h * hd;
        out[j * heads * hd + idx] = e < dim ? kn[j * heads * dim + (size_t)h * dim + e] : r[j * rot + (e - dim)];
    }
}

// scores [heads][rows][ld] (fp32, unscaled), heads head0, head0 + 1, ...  Row r belongs to position pos0 + r and sees keys 0 .. pos0 + r.  Its softmax
// (scores times scale, the sink in the denominator) is written as two bf16 numbers per weight, p = hi + lo, so that the
// product with the values keeps the weights' 32-bit precision in effect; keys out of sight get zeros.
__global__ void __launch_bounds__(256) softmax_split_kernel(const float* __restrict__ s, int ld, int rows, int n_pad, int pos0, float scale,
                                                            const void* sink, int sink_dtype, int head0, bf16* __restrict__ hi,
                                                            bf16* __restrict__ lo, int ld_p) {
    __shared__ float red[8];
    __shared__ float bc;
    fr_pdl_wait();
    fr_pdl_launch();
    const size_t row = blockIdx.x;
    const int head = head0 + (int)(row / rows), n = min(pos0 + (int)(row % rows) + 1, n_pad);
    const float* sr = s + row * ld;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float m = -INFINITY;
    for (int j = threadIdx.x; j < n; j += blockDim.x) m = fmaxf(m, sr[j] * scale);
    m = fr_warp_max(m);
    if (lane == 0) red[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = red[0];
        for (int i = 1; i < 8; ++i) t = fmaxf(t, red[i]);
        if (sink != nullptr) t = fmaxf(t, FrVec{sink, sink_dtype}.at(head));
        bc = t;
    }
    __syncthreads();
    m = bc;
    float l = 0.f;
    for (int j = threadIdx.x; j < n; j += blockDim.x) l += expf(sr[j] * scale - m);
    l = fr_warp_sum(l);
    __syncthreads();
    if (lane == 0) red[warp] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < 8; ++i) t += red[i];
        if (sink != nullptr) t += expf(FrVec{sink, sink_dtype}.at(head) - m);
        bc = 1.0f / t;
    }
    __syncthreads();
    const float inv = bc;
    bf16* h = hi + row * ld_p;
    bf16* o = lo + row * ld_p;
    for (int j = threadIdx.x; j < n_pad; j += blockDim.x) {
        const float p = j < n ? expf(sr[j] * scale - m) * inv : 0.f;
        const bf16 ph = __float2bfloat16_rn(p);
        h[j] = ph;
        o[j] = __float2bfloat16_rn(p - __bfloat162float(ph));
    }
}

// out[row][h * vd + n] = x[h][row][n] * sigmoid(gate[row][gate_off + h]) (gate null: 1), fp32 [heads][rows][vd] -> T [rows][heads * vd]
template <typename T>
__global__ void gate_cast_kernel(const float* __restrict__ x, const T* __restrict__ gate, int ld_gate, int gate_off, int heads, int vd,
                                 T* __restrict__ out) {
    fr_pdl_wait();
    fr_pdl_launch();
    const size_t row = blockIdx.x;
    for (int i = threadIdx.x; i < heads * vd; i += blockDim.x) {
        float v = x[((size_t)(i / vd) * gridDim.x + row) * vd + i % vd];
        if (gate != nullptr) v *= 1.0f / (1.0f + expf(-fr_load(gate + row * ld_gate + gate_off + i / vd)));
        fr_store(out + row * heads * vd + i, v);
    }
}

}  // namespace

FR_EXPORT int attention_latent_rotate_pairs(void* x, int ld, const int* row_seq, const int* row_pos, const float* freq, float mult,
                                            int rows, int heads, int head_stride, int first, int dims, int dtype,
                                            cudaStream_t stream) {
    if (rows <= 0 || heads <= 0 || dims <= 0) return FR_OK;
    if (dims % 2) FR_REFUSE("rotate_pairs: %d rotated dimensions (must be even)", dims);
    RotateArgs p{x, row_seq, row_pos, freq, mult, ld, rows, heads, head_stride, first, dims};
    if (dtype == FR_F32) FR_CUDA(fr_launch(rotate_pairs_kernel<float>, dim3(rows), dim3(128), 0, stream, p));
    else if (dtype == FR_BF16) FR_CUDA(fr_launch(rotate_pairs_kernel<bf16>, dim3(rows), dim3(128), 0, stream, p));
    else FR_REFUSE("rotate_pairs: unknown dtype %d", dtype);
    FR_CHECK_LAUNCH("rotate_pairs");
    return FR_OK;
}

FR_EXPORT int attention_latent_prepare(const void* x, int ld, int q_off, int kv_off, void* ckr, float* qf, const void* norm_w,
                                       int norm_dtype, float eps, const int* row_seq, const int* row_pos, const float* freq,
                                       float mult, int rows, int heads, int dim, int rot, int rot_dims, int rank, int dtype,
                                       cudaStream_t stream) {
    if (rows <= 0) return FR_OK;
    if (rot_dims % 2 || rot_dims < 0 || rot_dims > rot || rank <= 0 || heads <= 0)
        FR_REFUSE("latent prepare: rank %d, rotated part %d of which %d turn, %d heads", rank, rot, rot_dims, heads);
    PrepareArgs p{x, ckr, qf, norm_w, norm_dtype, row_seq, row_pos, freq, mult, eps, ld, q_off, kv_off, heads, dim, rot, rank, rot_dims};
    if (dtype == FR_F32) FR_CUDA(fr_launch(prepare_kernel<float>, dim3(rows), dim3(256), 0, stream, p));
    else if (dtype == FR_BF16) FR_CUDA(fr_launch(prepare_kernel<bf16>, dim3(rows), dim3(256), 0, stream, p));
    else FR_REFUSE("latent prepare: unknown dtype %d", dtype);
    FR_CHECK_LAUNCH("latent prepare");
    return FR_OK;
}

// Whether the products in 16-byte pieces are the faster form: up to a few rounds of blocks, where the chain of waits is the cost.
// Beyond, a block's set-up and its sums over the groups or lanes count (layout 0: until k is long, layout 1: where it is).  us, a column
// at a time / in pieces: layout 0, 16 x 24 2.5 / 2.8; 64 x 64, 64 rows x 32 heads 3.5 / 3.0, 300 x 32 9.8 / 22.9; 128 x 512, 31 x 32 1.2
// times as fast, 300 x 32 91 / 108; 256 x 512 1.03 to 3.2 times; layout 1, 64 x 64 1.2 to 2.8 times; 512 x 128, 64 x 32 1.0 times,
// 300 x 32 209 / 233.
static bool pieces_pay(int layout, int rows, int heads, int k, int n) {
    const long long blocks = (long long)((rows + HL_ROWS - 1) / HL_ROWS) * heads * (layout == 0 ? (n + 127) / 128 : (n + 15) / 16);
    if (layout == 0) return k >= 192 || (k >= 32 && blocks <= (long long)k * k / 12);
    return k <= 128 || blocks * k <= 1 << 20;
}

// x_dtype / w_dtype / out_dtype: FR_F32 or FR_BF16 each; the gate (if any) is stored in the result's dtype.
// fixed_weights not zero: w is memory that no kernel writes any more, and may be read while the kernel before still runs.
FR_EXPORT int attention_latent_head_linear_weights(const void* x, int x_dtype, int ld_x, int x_off, int x_stride, const void* w, int w_dtype,
                                                   int layout, void* out, int out_dtype, int ld_out, int out_stride, const void* gate,
                                                   int ld_gate, int gate_off, const int* row_seq, int rows, int heads, int k, int n,
                                                   int fixed_weights, cudaStream_t stream) {
    if (rows <= 0) return FR_OK;
    if (heads <= 0 || k <= 0 || n <= 0) FR_REFUSE("head_linear: %d heads, k %d, n %d", heads, k, n);
    HeadLinearArgs p{x, w, out, gate, row_seq, rows, heads, k, n, ld_x, x_off, x_stride, ld_out, out_stride, ld_gate, gate_off, fixed_weights};
    const int key = x_dtype * 4 + w_dtype * 2 + out_dtype;
    // bf16 weights whose rows (of n numbers in layout 0, of k in layout 1) are whole 16-byte pieces, where pieces_pay
    if (w_dtype == FR_BF16 && (layout == 0 ? n : k) % 8 == 0 && ((uintptr_t)w & 15) == 0 && (size_t)HL_ROWS * k * sizeof(float) <= 48 * 1024 &&
        pieces_pay(layout, rows, heads, k, n)) {
        if (key == 6) return launch_head_pieces<bf16, float>(p, layout, stream);
        if (key == 3) return launch_head_pieces<float, bf16>(p, layout, stream);
        if (key == 2) return launch_head_pieces<float, float>(p, layout, stream);
        if (key == 7) return launch_head_pieces<bf16, bf16>(p, layout, stream);
    }
    switch (key) {
        case 0: return launch_head_linear<float, float, float>(p, layout, stream);
        case 4 + 2 + 0: return launch_head_linear<bf16, bf16, float>(p, layout, stream);
        case 0 + 2 + 1: return launch_head_linear<float, bf16, bf16>(p, layout, stream);
        case 0 + 2 + 0: return launch_head_linear<float, bf16, float>(p, layout, stream);
        case 4 + 2 + 1: return launch_head_linear<bf16, bf16, bf16>(p, layout, stream);
        default: FR_REFUSE("head_linear: dtypes x %d, weights %d, out %d are not a combination that is built", x_dtype, w_dtype, out_dtype);
    }
}

// The same for weights that any earlier kernel of the stream may have made.
FR_EXPORT int attention_latent_head_linear(const void* x, int x_dtype, int ld_x, int x_off, int x_stride, const void* w, int w_dtype,
                                           int layout, void* out, int out_dtype, int ld_out, int out_stride, const void* gate,
                                           int ld_gate, int gate_off, const int* row_seq, int rows, int heads, int k, int n,
                                           cudaStream_t stream) {
    return attention_latent_head_linear_weights(x, x_dtype, ld_x, x_off, x_stride, w, w_dtype, layout, out, out_dtype, ld_out, out_stride,
                                                gate, ld_gate, gate_off, row_seq, rows, heads, k, n, 0, stream);
}

// Whether blocks with all heads of a row are the faster form.  Their time hardly depends on the heads (a warp has one of 1 to 8,
// two of 9 to 16, up to four of 17 to 32), that of a warp per head grows with them, and a block's rounds are a chain, so that few
// heads want few keys per block and several per warp many keys.  Latent 512 + 64, us, a warp per head / a block per row: 1 head, 8 rows x 2,000 keys 49 / 15,
// 64 x 2,000 116 / 159, 1,000 x 600 174 / 703; 4 heads, 64 x 2,000 1.1 times as fast, 256 x 600 173 / 204; 8 heads and 16: 1.0 to
// 3.8 times from 150 keys on, 8 rows x 20 keys 1.1 times and 10.1 / 12.8; 17 heads, 8 rows x 600 1.2 times, 64 x 600 176 / 237;
// 24 heads, 64 x 600 1.5 times, 256 x 600 0.95 times, 8 x 20 10.2 / 15.9.
static bool rows_pay(int rows, int heads, int keys) {
    if (heads <= 4) return rows <= 16 || (rows <= 256 && (long long)rows * keys <= (rows <= 64 ? 32768ll : 8192ll) * heads);
    if (heads <= 8) return rows <= 32 || keys >= 48;
    if (heads <= 16) return keys >= 4 * heads;
    return (rows <= 8 && keys >= 4 * heads) || (heads >= 22 && rows <= 64 && keys >= 256);
}

// Splits of the keys for a call of `rows` rows that see at most `keys`: two blocks per SM, at least one round of keys each; 0: not
// a call for the kernel whose blocks have all heads of a row (then a split is a warp's work).
FR_EXPORT int attention_latent_splits(int rows, int heads, int keys, int rank, int rot, int dtype) {
    if (rows <= 0 || !shared_rows(heads, rank, rot, dtype) || !rows_pay(rows, heads, keys)) return 0;
    const int sms = fr_sm_count() > 0 ? fr_sm_count() : 148;
    int splits = 2 * sms / rows;
    if (splits > (keys + KEYS - 1) / KEYS) splits = (keys + KEYS - 1) / KEYS;
    return splits < 1 ? 1 : splits;
}

// all_heads: blocks with all heads of a row, where the cache allows it (attention_latent_splits above 0 asks for it).
FR_EXPORT int attention_latent_form(const float* q, float* out, const void* c_pool, const void* r_pool, const int* block_table,
                                    int table_width, int page, const int* row_seq, const int* row_pos, const void* sink, int sink_dtype,
                                    int rows, int heads, int rank, int rot, float scale, int splits, float* scratch, int dtype,
                                    int all_heads, cudaStream_t stream) {
    if (rows <= 0) return FR_OK;
    if (rank <= 0 || rank > 32 * C_PER_LANE) FR_REFUSE("latent attention: latent size %d is outside 1..%d", rank, 32 * C_PER_LANE);
    if (rot < 0 || rot > 32 * R_PER_LANE) FR_REFUSE("latent attention: rotated part %d is outside 0..%d", rot, 32 * R_PER_LANE);
    if (splits < 1 || splits > 65535) FR_REFUSE("latent attention: %d splits", splits);
    if (splits > 1 && scratch == nullptr) FR_REFUSE("latent attention: splits need a scratch buffer");
    AttnArgs p{q, out, c_pool, r_pool, block_table, row_seq, row_pos, sink, sink_dtype, scratch, table_width, page, rows, heads, rank,
               rot, splits, scale};
    const int items = rows * heads;
    const dim3 grid((items + 3) / 4, splits);
    if (all_heads && shared_rows(heads, rank, rot, dtype) && (((uintptr_t)c_pool | (uintptr_t)r_pool) & 15) == 0) {
        if (heads <= 8) FR_CUDA(launch_rows<1>(p, stream));
        else if (heads <= 16) FR_CUDA(launch_rows<2>(p, stream));
        else FR_CUDA(launch_rows<4>(p, stream));
        FR_CHECK_LAUNCH("latent attention (shared rows)");
        if (splits > 1) {
            FR_CUDA(fr_launch(latent_merge_kernel, dim3(items), dim3(256), 0, stream, p));
            FR_CHECK_LAUNCH("latent attention merge");
        }
        return FR_OK;
    }
    const bool pairs = rank % 2 == 0 && rot % 2 == 0 && (((uintptr_t)c_pool | (uintptr_t)r_pool) & 7) == 0;
    if (dtype == FR_F32 && pairs) FR_CUDA(fr_launch(latent_attention_kernel<float, 2>, grid, dim3(128), 0, stream, p));
    else if (dtype == FR_F32) FR_CUDA(fr_launch(latent_attention_kernel<float, 1>, grid, dim3(128), 0, stream, p));
    else if (dtype == FR_BF16 && pairs) FR_CUDA(fr_launch(latent_attention_kernel<bf16, 2>, grid, dim3(128), 0, stream, p));
    else if (dtype == FR_BF16) FR_CUDA(fr_launch(latent_attention_kernel<bf16, 1>, grid, dim3(128), 0, stream, p));
    else FR_REFUSE("latent attention: unknown dtype %d", dtype);
    FR_CHECK_LAUNCH("latent attention");
    if (splits > 1) {
        FR_CUDA(fr_launch(latent_merge_kernel, dim3(items), dim3(256), 0, stream, p));
        FR_CHECK_LAUNCH("latent attention merge");
    }
    return FR_OK;
}

FR_EXPORT int attention_latent(const float* q, float* out, const void* c_pool, const void* r_pool, const int* block_table,
                               int table_width, int page, const int* row_seq, const int* row_pos, const void* sink, int sink_dtype,
                               int rows, int heads, int rank, int rot, float scale, int splits, float* scratch, int dtype,
                               cudaStream_t stream) {
    return attention_latent_form(q, out, c_pool, r_pool, block_table, table_width, page, row_seq, row_pos, sink, sink_dtype, rows, heads, rank,
                                 rot, scale, splits, scratch, dtype, 1, stream);
}

// One sequence's cached rows 0 .. n-1 (table: the sequence's row of the block table) as contiguous [2 n_pad][rank] (the
// latents twice, one below the other) and [n_pad][rot]; rows from n on are zero.
FR_EXPORT int attention_latent_gather(const void* c_pool, const void* r_pool, const int* table, int page, int n, int n_pad, int rank,
                                      int rot, void* c_all, void* r_all, int dtype, cudaStream_t stream) {
    if (n_pad <= 0) return FR_OK;
    if (dtype == FR_F32) FR_CUDA(fr_launch(gather_kernel<float>, dim3(n_pad), dim3(128), 0, stream, (const float*)c_pool, (const float*)r_pool, table, page, n, n_pad, rank, rot, (float*)c_all, (float*)r_all));
    else if (dtype == FR_BF16) FR_CUDA(fr_launch(gather_kernel<bf16>, dim3(n_pad), dim3(128), 0, stream, (const bf16*)c_pool, (const bf16*)r_pool, table, page, n, n_pad, rank, rot, (bf16*)c_all, (bf16*)r_all));
    else FR_REFUSE("latent gather: unknown dtype %d", dtype);
    FR_CHECK_LAUNCH("latent gather");
    return FR_OK;
}

// hi and lo: rows of ld_p numbers each (the two may be halves of one buffer's rows)
FR_EXPORT int attention_latent_softmax_split(const float* scores, int ld, int rows, int heads, int n_pad, int pos0, float scale, const void* sink,
                                             int sink_dtype, int head, void* hi, void* lo, int ld_p, cudaStream_t stream) {
    if (rows <= 0 || heads <= 0) return FR_OK;
    FR_CUDA(fr_launch(softmax_split_kernel, dim3((unsigned)((long long)rows * heads)), dim3(256), 0, stream, scores, ld, rows, n_pad, pos0, scale, sink, sink_dtype, head,
                      (bf16*)hi, (bf16*)lo, ld_p));
    FR_CHECK_LAUNCH("softmax_split");
    return FR_OK;
}

FR_EXPORT int attention_latent_gate_cast(const float* x, const void* gate, int ld_gate, int gate_off, int rows, int heads, int vd,
                                         void* out, int dtype, cudaStream_t stream) {
    if (rows <= 0) return FR_OK;
    if (dtype == FR_F32) FR_CUDA(fr_launch(gate_cast_kernel<float>, dim3(rows), dim3(256), 0, stream, x, (const float*)gate, ld_gate, gate_off, heads, vd, (float*)out));
    else if (dtype == FR_BF16) FR_CUDA(fr_launch(gate_cast_kernel<bf16>, dim3(rows), dim3(256), 0, stream, x, (const bf16*)gate, ld_gate, gate_off, heads, vd, (bf16*)out));
    else FR_REFUSE("gate_cast: unknown dtype %d", dtype);
    FR_CHECK_LAUNCH("gate_cast");
    return FR_OK;
}

FR_EXPORT int attention_latent_key_concat(const void* kn, const void* r, int rows, int heads, int dim, int rot, void* out, int dtype,
                                          cudaStream_t stream) {
    if (rows <= 0) return FR_OK;
    if (dtype == FR_F32) FR_CUDA(fr_launch(key_concat_kernel<float>, dim3(rows), dim3(256), 0, stream, (const float*)kn, (const float*)r, heads, dim, rot, (float*)out));
    else if (dtype == FR_BF16) FR_CUDA(fr_launch(key_concat_kernel<bf16>, dim3(rows), dim3(256), 0, stream, (const bf16*)kn, (const bf16*)r, heads, dim, rot, (bf16*)out));
    else FR_REFUSE("key_concat: unknown dtype %d", dtype);
    FR_CHECK_LAUNCH("key_concat");
    return FR_OK;
}
