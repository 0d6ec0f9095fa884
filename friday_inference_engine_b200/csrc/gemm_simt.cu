// out[m][n] = sum_k a[m][k] * w[n][k]  (+ bias[n]) (+ residual[m][n])
//
// Matrix product with fp32 multiply-adds: the true 32-bit path of the model (no
// reduced-precision mode; many rows go to gemm_f32_tc.cuh, which keeps the operands'
// 24 bits), and the fallback of the bf16 path for sizes that the tensor-core
// kernel refuses.  Both operands are row-major with k
// innermost, which is how activations [rows][k] and projection weights [out][in] are
// stored, so nothing is transposed.  Any m, n, k.  Four kernels:
//
//   gemm_f32_kernel    fp32 operands in 16-byte pieces, more rows than the next one takes:
//                      tiles in registers, k in two interleaved sums (fma.rn.f32x2), k split
//                      over the CTAs of a cluster where there are few tiles;
//   few_rows_kernel    the same operands, up to FEW_ROWS rows (FEW_ROWS_WIDE from 8,192
//                      columns on): a warp per few columns, its lanes along k;
//   few_fused_kernel   the same with its neighbours' work at both ends (gemm_few_fusion.h);
//   gemm_simt_kernel   everything else (mixed storage, unaligned rows).
//
// The reference's counterpart is its int8 tensor-core GEMM with the same epilogue
// (bias, then residual, in place allowed): prefill_kernels.cu:156-171, 173-327.
#include "gemm_f32_tc.cuh"
#include "gemm_few_fusion.h"

FR_EXPORT const char* gemm_simt_last_error() { return fr_error_text; }

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;   // 256 threads, 4x4 outputs each

template <typename TA, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ a, const TW* __restrict__ w, TO* out, FrVec bias, const TO* residual, int m,
                 int n, int k, int lda, int ldw, int ldo) {
    __shared__ float as[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;     // tx: 4 columns, ty: 4 rows
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < k; k0 += BK) {
        // 64 x 16 elements per operand, 4 per thread; consecutive threads read consecutive k.
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int idx = tid + r * 256;
            const int row = idx / BK, kk = idx % BK;
            const int gk = k0 + kk;
            float va = 0.f, vw = 0.f;
            if (gk < k) {
                if (m0 + row < m) va = fr_load(a + (size_t)(m0 + row) * lda + gk);
                if (n0 + row < n) vw = fr_load(w + (size_t)(n0 + row) * ldw + gk);
            }
            as[kk][row] = va;
            ws[kk][row] = vw;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float ra[TM], rw[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) ra[i] = as[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) rw[j] = ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(ra[i], rw[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= m) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn >= n) continue;
            float v = acc[i][j];
            if (bias.p != nullptr) v += bias.at(gn);
            if (residual != nullptr) v += fr_load(residual + (size_t)gm * ldo + gn);
            fr_store(out + (size_t)gm * ldo + gn, v);
        }
    }
}

template <typename TA, typename TW, typename TO>
int launch(const void* a, const void* w, void* out, FrVec bias, const void* residual, int m, int n, int k, int lda,
           int ldw, int ldo, cudaStream_t stream) {
    dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
    gemm_simt_kernel<TA, TW, TO><<<grid, 256, 0, stream>>>((const TA*)a, (const TW*)w, (TO*)out, bias,
                                                          (const TO*)residual, m, n, k, lda, ldw, ldo);
    FR_CHECK_LAUNCH("gemm_simt");
    return FR_OK;
}


// ------------------------------------------------------------------ fp32 operands in 16-byte pieces
typedef unsigned long long Pair;                            // two floats: the sums over k = 0, 2, ... and 1, 3, ...
__device__ __forceinline__ void fma_pair(Pair& acc, Pair x, Pair y) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y)); }
__device__ __forceinline__ float pair_sum(Pair v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }

struct F32Args {
    const float* a;
    const float* w;
    float* out;
    FrVec bias;
    const float* residual;
    int m, n, k, lda, ldw, ldo;
    int splits, kb_per;          // CTAs of the cluster that share a tile's k, k blocks of each
    int fixed_weights;           // no kernel writes them any more: they may be read ahead of the wait for the kernel before
};

__device__ __forceinline__ void finish(const F32Args& p, int gm, int gn, float v) {
    if (gm >= p.m || gn >= p.n) return;
    if (p.bias.p != nullptr) v += p.bias.at(gn);
    const size_t at = (size_t)gm * p.ldo + gn;
    if (p.residual != nullptr) v += p.residual[at];
    p.out[at] = v;
}

constexpr int F32_BK = 32, F32_LD = F32_BK + 4, F32_STAGES = 3;   // LD: eight consecutive rows' 16-byte pieces lie in different banks
template <int TM, int TN>
constexpr int f32_smem() { return F32_STAGES * (8 * TM + 16 * TN) * F32_LD * 4; }

// 128 threads, 8 TM x 16 TN outputs, TM x TN per thread: a warp has 4 rows x 8 columns of threads, whose rows and columns lie
// 4 and 8 apart.  Both operands keep their k-innermost layout in shared memory, so that a 16-byte read gives two operand pairs
// of the packed multiply-add as they are; the two halves of an accumulator are added at the end.  Bound by the rate of the
// multiply-adds: per 4 k a warp issues 2 TM TN of them (two cycles each) and TM + TN shared-memory reads.
template <int TM, int TN>
__global__ void __launch_bounds__(128, 2)
gemm_f32_kernel(const F32Args p) {
    constexpr int BM = 8 * TM, BN = 16 * TN, STAGE = (BM + BN) * F32_LD;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x / p.splits, split = blockIdx.x - tile * p.splits;
    const int m0 = blockIdx.y * BM, n0 = tile * BN;
    const int kb0 = split * p.kb_per, kb1 = min((p.k + F32_BK - 1) / F32_BK, kb0 + p.kb_per);
    // neighbouring lanes share a column, so that both operands of a half-warp take one pass through the banks
    const int row0 = (warp >> 1) * 4 * TM + (lane >> 4) * 2 + (lane & 1), col0 = (warp & 1) * 8 * TN + ((lane >> 1) & 7);
    fr_pdl_wait();
    fr_pdl_launch();
    auto fill = [&](int kb, int stage) {
        float* base = sm + stage * STAGE;
#pragma unroll
        for (int i = 0; i < (BM + BN + 15) / 16; ++i) {
            const int idx = tid + i * 128, r = idx >> 3, c = (idx & 7) * 4;
            if ((BM + BN) % 16 != 0 && r >= BM + BN) break;
            const int gk = kb * F32_BK + c;
            const bool of_a = r < BM;
            const int g = of_a ? m0 + r : n0 + r - BM;
            const bool there = gk < p.k && g < (of_a ? p.m : p.n);
            const float* src = there ? (of_a ? p.a + (size_t)g * p.lda + gk : p.w + (size_t)g * p.ldw + gk) : p.w;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(base + r * F32_LD + c)),
                         "l"(src), "r"(there ? 16 : 0)
                         : "memory");
        }
    };
    Pair acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int s = 0; s < F32_STAGES - 1; ++s) {
        if (kb0 + s < kb1) fill(kb0 + s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
        asm volatile("cp.async.wait_group %0;" ::"n"(F32_STAGES - 2) : "memory");
        __syncthreads();                                     // this block is here, and everyone is done with the one before
        const int refill = stage == 0 ? F32_STAGES - 1 : stage - 1;
        if (kb + F32_STAGES - 1 < kb1) fill(kb + F32_STAGES - 1, refill);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = sm + stage * STAGE + row0 * F32_LD;
        const float* ws = sm + stage * STAGE + (BM + col0) * F32_LD;
#pragma unroll
        for (int kk = 0; kk < F32_BK; kk += 4) {
            ulonglong2 x[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) x[i] = *(const ulonglong2*)(as + i * 4 * F32_LD + kk);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 y = *(const ulonglong2*)(ws + j * 8 * F32_LD + kk);
#pragma unroll
                for (int i = 0; i < TM; ++i) fma_pair(acc[i][j], x[i].x, y.x);
#pragma unroll
                for (int i = 0; i < TM; ++i) fma_pair(acc[i][j], x[i].y, y.y);
            }
        }
        if (++stage == F32_STAGES) stage = 0;
    }
    if (p.splits == 1) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) finish(p, m0 + row0 + 4 * i, n0 + col0 + 8 * j, pair_sum(acc[i][j]));
        return;
    }
    // the tile's parts lie in the shared memory of the cluster's CTAs; each finishes a share of it, adding them in order of k
    static_assert(BM * BN <= F32_STAGES * STAGE, "the partial tile takes the ring's place");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sm[(row0 + 4 * i) * BN + col0 + 8 * j] = pair_sum(acc[i][j]);
    fr_cluster_sync();
    for (int idx = (split * 128 + tid) * 4; idx < BM * BN; idx += p.splits * 512) {
        float4 v = fr_cluster_load4(sm + idx, 0);
        for (int s = 1; s < p.splits; ++s) {
            const float4 o = fr_cluster_load4(sm + idx, s);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        const int gm = m0 + idx / BN, gn = n0 + idx % BN;
        finish(p, gm, gn, v.x);
        finish(p, gm, gn + 1, v.y);
        finish(p, gm, gn + 2, v.z);
        finish(p, gm, gn + 3, v.w);
    }
    fr_cluster_sync();                                       // nobody leaves while its shared memory is being read
}

// Bound by reading the weights once (or by the launch, for small ones).  Up to MR rows per block: a warp has NC columns, its lanes
// take 16-byte pieces of k in turn, every weight is read once per block of rows; the MR * NC sums are then added over the lanes so
// that lane l ends with the l-th.
// Four columns per warp where there are enough of them to keep the SMs' loads in flight: a piece of x is then read once for
// four weights (4 x 37888 x 3584: 108 us, 5.0 TB/s, against 129 with one column; 2 x 5000 x 3584 22 us either way).  Against
// the general kernel: 694 and 338 us.  At 9 to 16 rows the weights are read twice, the second time from L2: up to 8,191
// columns that beats the tiles (12 x 3584 x 3584: 30 us against 38, 16 x 4608 x 3584: 35 against 44), above it does not
// (12 x 37888 x 3584: 212 us on tiles, the fastest form).
constexpr int FEW_ROWS = 16, FEW_ROWS_WIDE = 8;
template <int MR, int NC>
__global__ void __launch_bounds__(128)
few_rows_kernel(const F32Args p) {
    constexpr int V = MR * NC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (blockIdx.x * 4 + warp) * NC, m0 = blockIdx.y * MR;
    if (n0 >= p.n) {
        fr_pdl_wait();                                       // (no kernel ends before its predecessor)
        return;
    }
    Pair acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0ull;
    const ulonglong2* w[NC];
    const ulonglong2* x[MR];
#pragma unroll
    for (int c = 0; c < NC; ++c) w[c] = (const ulonglong2*)(p.w + (size_t)min(n0 + c, p.n - 1) * p.ldw);
#pragma unroll
    for (int r = 0; r < MR; ++r) x[r] = (const ulonglong2*)(p.a + (size_t)min(m0 + r, p.m - 1) * p.lda);
    // the first piece of fixed weights, which do not depend on the kernel before this one, ahead of the wait for it
    if (!p.fixed_weights) fr_pdl_wait();
    ulonglong2 first[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) first[c] = lane < p.k / 4 ? __ldg(w[c] + lane) : make_ulonglong2(0, 0);
    fr_pdl_wait();
    fr_pdl_launch();
#pragma unroll 2
    for (int q = lane; q < p.k / 4; q += 32) {
        ulonglong2 y[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) y[c] = q == lane ? first[c] : __ldg(w[c] + q);
#pragma unroll
        for (int r = 0; r < MR; ++r) {
            const ulonglong2 z = x[r][q];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                fma_pair(acc[r * NC + c], z.x, y[c].x);
                fma_pair(acc[r * NC + c], z.y, y[c].y);
            }
        }
    }
    float s[V];
#pragma unroll
    for (int v = 0; v < V; ++v) s[v] = pair_sum(acc[v]);
    // halve the values and double the lanes behind each: the half that a lane keeps is chosen by one of its bits
    int at = 0;
#pragma unroll
    for (int half = V / 2, bit = 16; bit > 0; bit >>= 1) {
        if (half > 0) {
            const bool upper = (lane & bit) != 0;
#pragma unroll
            for (int v = 0; v < V / 2; ++v)
                if (v < half) {
                    const float give = upper ? s[v] : s[v + half], keep = upper ? s[v + half] : s[v];
                    s[v] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            if (upper) at += half;
            half >>= 1;
        } else {
            s[0] += __shfl_xor_sync(0xffffffffu, s[0], bit);
        }
    }
    constexpr int SPARE = 32 / V;                            // lanes with the same value
    if (lane % SPARE == 0) finish(p, m0 + at / NC, n0 + at % NC, s[0]);
}

template <int MR, int NC>
int launch_few(const F32Args& p, cudaStream_t stream) {
    FR_CUDA(fr_launch(few_rows_kernel<MR, NC>, dim3((p.n + 4 * NC - 1) / (4 * NC), (p.m + MR - 1) / MR), dim3(128), 0, stream, p));
    FR_CHECK_LAUNCH("gemm_simt (few rows)");
    return FR_OK;
}

// The same with work of its neighbours at both ends (gemm_few_fusion.h).  A warp has NP pairs of columns: the two that a gated unit or a
// rotation needs lie in one warp.  The norm of the input is finished after the sums: every warp reads all of its rows anyway and
// adds up their squares on the way.
enum FewEnd { FEW_PLAIN, FEW_GATED, FEW_ROTARY };

// Columns of pair `pair` of a rotary product: (i, i + rot / 2) of a rotated head, neighbours elsewhere.
__device__ __forceinline__ void rotary_columns(const GemmFewFusion& f, int pair, int& c0, int& c1, int& head, int& angle) {
    const int per = f.hd >> 1;
    head = pair / per;
    const int i = pair - head * per, base = head * f.hd, half = f.rot >> 1;
    angle = -1;
    if (f.denom != nullptr && head < f.nq + f.nkv) {
        if (i < half) {
            angle = i;
            c0 = base + i;
            c1 = c0 + half;
            return;
        }
        c0 = base + f.rot + 2 * (i - half);
    } else {
        c0 = base + 2 * i;
    }
    c1 = c0 + 1;
}

// Bound by its launch, then by reading the weights.  4 x 160 x 96 with norm, rotation and cache write: 2.6 us in place of a chain of
// 2.1 (norm), 1.6 and 2.0 (rotation, store); 4 x 512 x 96 with norm and gated unit: 2.3 in place of 2.1, 1.6 and 1.2.  A prompt and
// sixteen tokens of such a model of three layers: 1,401 -> 1,246 us.
template <int MR, int NP, int END>
__global__ void __launch_bounds__(128)
few_fused_kernel(const F32Args p, const GemmFewFusion f) {
    constexpr int NC = 2 * NP, V = MR * NC, SPARE = 32 / V;
    static_assert(V <= 32, "a lane ends with one value");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pair0 = (blockIdx.x * 4 + warp) * NP, m0 = blockIdx.y * MR, pairs = (p.n + 1) >> 1;
    if (pair0 >= pairs) {
        fr_pdl_wait();                                       // (no kernel ends before its predecessor)
        return;
    }
    int col[NC];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const int pair = min(pair0 + q, pairs - 1);
        int head, angle;
        if (END == FEW_ROTARY) {
            rotary_columns(f, pair, col[2 * q], col[2 * q + 1], head, angle);
        } else {
            col[2 * q] = 2 * pair;
            col[2 * q + 1] = min(2 * pair + 1, p.n - 1);
        }
    }
    // what this lane finishes: value `at` of row m0 + at / NC and column at % NC of the warp's
    const int at = lane / SPARE, my_row = m0 + at / NC, my_pair = pair0 + (at % NC) / 2, second = at & 1;
    // its angle and cache row depend on the step's geometry alone
    float cosine = 1.f, sine = 0.f;
    float* cached = nullptr;
    if (END == FEW_ROTARY && my_row < p.m && my_pair < pairs && f.row_seq[my_row] >= 0) {
        int c0, c1, head, angle;
        rotary_columns(f, my_pair, c0, c1, head, angle);
        const int pos = f.row_pos[my_row];
        if (angle >= 0) sincosf(__fdiv_rn((float)pos, f.denom[angle]), &sine, &cosine);
        if (f.k_pool != nullptr && head >= f.nq) {
            const int page = f.table[(size_t)f.row_seq[my_row] * f.table_width + pos / f.page];
            const bool is_k = head < f.nq + f.nkv;
            cached = (is_k ? f.k_pool : f.v_pool) + (((size_t)page * f.page + pos % f.page) * f.nkv + (head - f.nq - (is_k ? 0 : f.nkv))) * f.hd +
                     (second ? c1 : c0) - head * f.hd;
        }
    }
    const FrVec gain{f.norm_w, f.norm_w_dtype};
    Pair acc[V];
    float squares[MR];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0ull;
#pragma unroll
    for (int r = 0; r < MR; ++r) squares[r] = 0.f;
    const ulonglong2* w[NC];
    const float4* x[MR];
#pragma unroll
    for (int c = 0; c < NC; ++c) w[c] = (const ulonglong2*)(p.w + (size_t)col[c] * p.ldw);
#pragma unroll
    for (int r = 0; r < MR; ++r) x[r] = (const float4*)(p.a + (size_t)min(m0 + r, p.m - 1) * p.lda);
    if (!p.fixed_weights) fr_pdl_wait();
    ulonglong2 first[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) first[c] = lane < p.k / 4 ? __ldg(w[c] + lane) : make_ulonglong2(0, 0);
    fr_pdl_wait();
    fr_pdl_launch();
#pragma unroll 2
    for (int q = lane; q < p.k / 4; q += 32) {
        ulonglong2 y[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) y[c] = q == lane ? first[c] : __ldg(w[c] + q);
        float g[4] = {1.f, 1.f, 1.f, 1.f};
        if (f.norm_w != nullptr) gain.four(4 * q, g);
#pragma unroll
        for (int r = 0; r < MR; ++r) {
            float4 z = x[r][q];
            if (f.norm_w != nullptr) {
                squares[r] = fmaf(z.x, z.x, fmaf(z.y, z.y, fmaf(z.z, z.z, fmaf(z.w, z.w, squares[r]))));
                z.x *= g[0]; z.y *= g[1]; z.z *= g[2]; z.w *= g[3];
            }
            const Pair lo = (Pair)__float_as_uint(z.x) | (Pair)__float_as_uint(z.y) << 32;
            const Pair hi = (Pair)__float_as_uint(z.z) | (Pair)__float_as_uint(z.w) << 32;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                fma_pair(acc[r * NC + c], lo, y[c].x);
                fma_pair(acc[r * NC + c], hi, y[c].y);
            }
        }
    }
    float s[V];
#pragma unroll
    for (int v = 0; v < V; ++v) s[v] = pair_sum(acc[v]);
    if (f.norm_w != nullptr) {
#pragma unroll
        for (int r = 0; r < MR; ++r) {
            const float inv = 1.0f / sqrtf(fr_warp_sum(squares[r]) / (float)p.k + f.eps);
#pragma unroll
            for (int c = 0; c < NC; ++c) s[r * NC + c] *= inv;
        }
    }
#pragma unroll
    for (int half = V / 2, bit = 16; bit > 0; bit >>= 1) {     // as in few_rows_kernel: lane l ends with value l / SPARE
        if (half > 0) {
            const bool upper = (lane & bit) != 0;
#pragma unroll
            for (int v = 0; v < V / 2; ++v)
                if (v < half) {
                    const float give = upper ? s[v] : s[v + half], keep = upper ? s[v + half] : s[v];
                    s[v] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            half >>= 1;
        } else {
            s[0] += __shfl_xor_sync(0xffffffffu, s[0], bit);
        }
    }
    int c0 = 2 * my_pair, c1 = c0 + 1, head = 0, angle = -1;
    if (END == FEW_ROTARY && my_pair < pairs) rotary_columns(f, my_pair, c0, c1, head, angle);
    const int my_col = second ? c1 : c0;
    const bool mine = lane % SPARE == 0 && my_row < p.m && my_pair < pairs && my_col < p.n;
    float v = s[0];
    if (mine && p.bias.p != nullptr) v += p.bias.at(my_col);
    const float other = __shfl_xor_sync(0xffffffffu, v, SPARE);
    if (!mine) return;
    if (END == FEW_GATED) {
        if (!second) p.out[(size_t)my_row * p.ldo + my_pair] = fr_gated(f.act, v, other, f.act_limit, f.act_slope);
    } else {
        if (END == FEW_ROTARY && angle >= 0 && f.row_seq[my_row] >= 0) {
            float ra, rb;
            fr_rotate(second ? other : v, second ? v : other, cosine, sine, ra, rb);
            v = second ? rb : ra;
        }
        const size_t to = (size_t)my_row * p.ldo + my_col;
        if (p.residual != nullptr) v += p.residual[to];
        p.out[to] = v;
        if (END == FEW_ROTARY && cached != nullptr) *cached = v;
    }
}

template <int MR, int NP>
int launch_few_fused(const F32Args& p, const GemmFewFusion& f, cudaStream_t stream) {
    const dim3 grid(((p.n + 1) / 2 + 4 * NP - 1) / (4 * NP), (p.m + MR - 1) / MR);
    if (f.nq > 0) FR_CUDA(fr_launch(few_fused_kernel<MR, NP, FEW_ROTARY>, grid, dim3(128), 0, stream, p, f));
    else if (f.act) FR_CUDA(fr_launch(few_fused_kernel<MR, NP, FEW_GATED>, grid, dim3(128), 0, stream, p, f));
    else FR_CUDA(fr_launch(few_fused_kernel<MR, NP, FEW_PLAIN>, grid, dim3(128), 0, stream, p, f));
    FR_CHECK_LAUNCH("gemm_simt (few rows, fused)");
    return FR_OK;
}

template <int TM, int TN>
int launch_f32(const F32Args& p, cudaStream_t stream) {
    static std::atomic<unsigned long long> configured{0};    // devices (as bits) on which the limit has been raised
    int device = 0;
    FR_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= 64) FR_REFUSE("gemm_simt: device %d is outside the table of 64", device);
    if (!(configured.load(std::memory_order_acquire) & (1ull << device))) {
        FR_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_smem<TM, TN>()));
        configured.fetch_or(1ull << device, std::memory_order_release);
    }
    const dim3 grid((p.n + 16 * TN - 1) / (16 * TN) * p.splits, (p.m + 8 * TM - 1) / (8 * TM));
    FR_CUDA(fr_launch_cluster(gemm_f32_kernel<TM, TN>, grid, dim3(128), f32_smem<TM, TN>(), stream, (unsigned)p.splits, p));
    FR_CHECK_LAUNCH("gemm_simt (fp32)");
    return FR_OK;
}

// Tile and split of k: the choice whose busiest SM has the least to do (a lone CTA leaves a third of the multiply-add rate).  The
// cost of a k block is its multiply-adds, tm * tn, and 8 for what goes with them whatever the tile (barrier, copies, addresses); a
// CTA's start and end count as four blocks of the largest tile, a cluster's exchange as four more.  These weights only rank the
// choices; over 267 shapes (1 to 1,500 rows) the choice was never slower than the general kernel.
// Measured on B200, this kernel against the general one below: 333 x 37888 x 3584 1,902 us (47.6 TFLOP/s; two thirds of the
// rate at 1.88 GHz, whatever the tile and with plain multiply-adds too) against 3,998, 333 x 3584 x 18944 1,070 (7 x 8, four
// splits) against 2,923, 64 x 3584 x 3584 57 against 338, 40 x 3584 x 18944 164 against 3,133.
struct F32Plan {
    int tm, tn, splits;
};
F32Plan f32_plan(int m, int n, int k, int sms) {
    F32Plan best{8, 8, 1};
    double best_cost = 1e300;
    const int kb = (k + F32_BK - 1) / F32_BK;
    for (int tn = 8; tn >= 4; tn -= 4)
        for (int tm = 8; tm >= 4; --tm) {
            const long long tiles = (long long)((m + 8 * tm - 1) / (8 * tm)) * ((n + 16 * tn - 1) / (16 * tn));
            for (int s = 1; s <= 8; ++s) {
                if (s > 1 && kb < 4 * s) break;
                if (s > 2 && s != 4 && tiles * s > sms) continue;      // several waves of clusters of other sizes leave places empty
                const int per = (kb + s - 1) / s;
                const long long load = (tiles * s + sms - 1) / sms;
                const double block = tm * tn + 8.0;           // a k block's multiply-adds and what goes with them
                const double cost = (load == 1 ? 1.5 : (double)load) * (per * block + 4 * 64.0 + (s > 1 ? 4 * 64.0 : 0.0));
                if (cost < best_cost) { best_cost = cost; best = F32Plan{tm, tn, s}; }
            }
        }
    return best;
}

int run_f32(F32Args p, cudaStream_t stream) {
    if (p.m <= (p.n < 8192 ? FEW_ROWS : FEW_ROWS_WIDE)) {
        const bool wide = p.n >= 2368;
        if (p.m == 1) return wide ? launch_few<1, 4>(p, stream) : launch_few<1, 1>(p, stream);
        if (p.m == 2) return wide ? launch_few<2, 4>(p, stream) : launch_few<2, 1>(p, stream);
        if (p.m <= 4) return wide ? launch_few<4, 4>(p, stream) : launch_few<4, 1>(p, stream);
        return wide ? launch_few<8, 4>(p, stream) : launch_few<8, 1>(p, stream);
    }
    const int sms = fr_sm_count();
    const F32Plan plan = f32_plan(p.m, p.n, p.k, sms > 0 ? sms : 148);
    const int kb = (p.k + F32_BK - 1) / F32_BK;
    p.splits = plan.splits;
    p.kb_per = (kb + p.splits - 1) / p.splits;
#define FR_TILE(TM, TN) if (plan.tm == TM && plan.tn == TN) return launch_f32<TM, TN>(p, stream)
    FR_TILE(8, 8); FR_TILE(7, 8); FR_TILE(6, 8); FR_TILE(5, 8); FR_TILE(4, 8);
    FR_TILE(8, 4); FR_TILE(7, 4); FR_TILE(6, 4); FR_TILE(5, 4); FR_TILE(4, 4);
#undef FR_TILE
    FR_REFUSE("gemm_simt: no tile of %d x %d", plan.tm, plan.tn);
}

}  // namespace

// a: [m][k] (row stride lda), w: [n][k] (row stride ldw), out and residual: [m][n]
// (row stride ldo; residual may be `out` itself).  bias may be null; its dtype is
// given apart from the others because a bias stored in 32-bit stays so.
// fixed_weights not zero: w is memory that no kernel writes any more, and may be read while the kernel before still runs.
FR_EXPORT int gemm_simt_weights(const void* a, int a_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                                const void* bias, int bias_dtype, const void* residual, int m, int n, int k, int lda,
                                int ldw, int ldo, int fixed_weights, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return FR_OK;
    if (k <= 0) FR_REFUSE("gemm_simt: k = %d", k);
    FrVec bv{bias, bias_dtype};
    typedef __nv_bfloat16 bf16;
    // rows in 16-byte pieces (and no grid beyond the launch limits): the fp32 kernels
    if (a_dtype == FR_F32 && w_dtype == FR_F32 && out_dtype == FR_F32 && !((k | lda | ldw) & 3) && !(((uintptr_t)a | (uintptr_t)w) & 15) &&
        m <= 65535 * 32)
        return run_f32(F32Args{(const float*)a, (const float*)w, (float*)out, bv, (const float*)residual, m, n, k, lda, ldw, ldo, 1, 0, fixed_weights}, stream);
    const int key = a_dtype * 4 + w_dtype * 2 + out_dtype;
    switch (key) {
        case 0: return launch<float, float, float>(a, w, out, bv, residual, m, n, k, lda, ldw, ldo, stream);
        case 4: return launch<bf16, float, float>(a, w, out, bv, residual, m, n, k, lda, ldw, ldo, stream);
        case 5: return launch<bf16, float, bf16>(a, w, out, bv, residual, m, n, k, lda, ldw, ldo, stream);
        case 6: return launch<bf16, bf16, float>(a, w, out, bv, residual, m, n, k, lda, ldw, ldo, stream);
        case 7: return launch<bf16, bf16, bf16>(a, w, out, bv, residual, m, n, k, lda, ldw, ldo, stream);
        default: FR_REFUSE("gemm_simt: no kernel for dtypes a=%d w=%d out=%d", a_dtype, w_dtype, out_dtype);
    }
}

// The same for weights that any earlier kernel of the stream may have made.
FR_EXPORT int gemm_simt(const void* a, int a_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                        const void* bias, int bias_dtype, const void* residual, int m, int n, int k, int lda,
                        int ldw, int ldo, cudaStream_t stream) {
    return gemm_simt_weights(a, a_dtype, w, w_dtype, out, out_dtype, bias, bias_dtype, residual, m, n, k, lda, ldw, ldo, 0, stream);
}

// Products of fp32 operands on the tensor cores (gemm_f32_tc.cuh): whether gemm_simt_split takes this one with `scratch_bytes` of
// scratch, and is the faster way.  It has two launches and a longer chain from its first load to its last store: below some 2^20
// weights, or short k, the kernels of one launch are ahead (1024 x 512: 48 rows 10 us against 16; 1024 x 1024: 64 rows level, 128 rows
// 21 against 16; 2048 x 1024: 48 rows 17 against 14; 200000 x 64: 96 rows 74 against 88).  Fewer than four tiles of columns leave most
// SMs idle whatever the split of k (128 x 18944: 128 rows 47 against 51, 1,024 rows, in six portions, 214 against 343; 300 x 4096: 65 rows 12.7
// against 15.2, 333 rows 54 against 20).
// Rows beyond what the scratch holds go in portions, each of which reads and splits the weights again: with 38.8 MB, 341 rows of k = 18,944 at a
// time and 1,800 of 3,584 (3584 x 18944: 342 rows 216 us, 353 rows 288; the tiles of one launch take 1,280).
FR_EXPORT int gemm_simt_split_pays(const void* a, const void* w, int m, int n, int k, int lda, int ldw, long long scratch_bytes) {
    if (((k | lda | ldw) & 3) || (((uintptr_t)a | (uintptr_t)w) & 15) || k < 1024 || n < 256) return 0;
    const bool few = m <= (n < 8192 ? FEW_ROWS : FEW_ROWS_WIDE);
    const int at_once = split_rows_at_once(m, k, scratch_bytes);
    if (few || at_once == 0) return 0;
    if (n < 512 && (m < 160 || at_once < m)) return 0;
    const long long weights = (long long)n * k;
    return weights >= 2ll << 20 ? m >= 48 || weights >= 6ll << 20 : weights >= 1ll << 20 && m > (n >= 1024 ? 64 : 127);
}

// Kernels that gemm_simt_split launches: two per portion of rows.
FR_EXPORT int gemm_simt_split_launches(int m, int k, long long scratch_bytes) {
    const int rows = m > 0 && k > 0 ? split_rows_at_once(m, k, scratch_bytes) : 0;
    return rows > 0 ? 2 * ((m + rows - 1) / rows) : 0;
}

// scratch: 16-byte aligned, used by the kernels of this call only; status: a word that a wait that gave up is noted in.
FR_EXPORT int gemm_simt_split(const float* a, const float* w, float* out, const void* bias, int bias_dtype, const float* residual, int m, int n,
                              int k, int lda, int ldw, int ldo, int fixed_weights, void* scratch, long long scratch_bytes, int* status,
                              cudaStream_t stream) {
    if (m <= 0 || n <= 0) return FR_OK;
    if (k <= 0) FR_REFUSE("gemm_simt: k = %d", k);
    if (((k | lda | ldw) & 3) || (((uintptr_t)a | (uintptr_t)w | (uintptr_t)scratch) & 15)) FR_REFUSE("gemm_simt: rows are not in 16-byte pieces");
    const int rows = split_rows_at_once(m, k, scratch_bytes);
    if (rows == 0) FR_REFUSE("gemm_simt: %lld bytes of scratch are too few for rows of %d", scratch_bytes, k);
    for (int r0 = 0; r0 < m; r0 += rows) {
        const SplitArgs p{a + (size_t)r0 * lda, w, out + (size_t)r0 * ldo, FrVec{bias, bias_dtype}, residual ? residual + (size_t)r0 * ldo : nullptr,
                          nullptr, m - r0 < rows ? m - r0 : rows, n, k, lda, ldw, ldo, 0, 0, 0, 1, 0, fixed_weights, status};
        const int rc = run_split(p, scratch, stream);
        if (rc) return rc;
    }
    return FR_OK;
}

// Whether gemm_simt_few takes these rows and weights (as gemm_simt's kernel of few rows does).
FR_EXPORT int gemm_simt_few_supports(const float* a, const float* w, int m, int n, int k, int lda, int ldw) {
    return k > 0 && n > 0 && !((k | lda | ldw) & 3) && !(((uintptr_t)a | (uintptr_t)w) & 15) && m <= (n < 8192 ? FEW_ROWS : FEW_ROWS_WIDE);
}

// Whether gemm_simt_few is the faster way: `end` 0 a product alone, 1 a gated unit, 2 rotary columns; `norm`: with the norm of its input.  It saves
// the launches of its neighbours, 1 to 2 us each, and pays for them in the product itself: a third more registers, so fewer loads in flight, and
// the norm's multiplications in every warp.  Measured on B200 with the norm, us, the kernels one after another and this one:
//   one row: always ahead (4608 x 3584 rotary 42 and 21, 160 x 96 plain 3.0 and 1.8; 32768 x 96 plain 4.6 and 4.7)
//   two rows: up to 9472 columns (more do not fit the SMs at once: 9728 x 896 plain 10.7 and 13.4) and, if not rotary, k below 4096 (4608 x 3584
//   plain 27 and 22; 1024 x 4096 plain 22.7 and 24.1)
//   three and four: rotary up to 6144 columns (4608 x 3584 32 and 27; 8192 x 1024 14 and 19), gated up to 8192 columns of k up to 1024 (4864 x 896
//   10.1 and 8.8; 2048 x 2048 15 and 19), plain of k up to 128 (1000 x 96 3.2 and 2.6; 512 x 256 3.4 and 3.7)
//   five to sixteen: gated and rotary up to 1024 x 512, with a norm (512 x 96 gated 4.3 and 3.4; 8 x 4608 x 3584 rotary 37 and 53, 16 rows 56 and 143)
FR_EXPORT int gemm_simt_few_pays(int m, int n, int k, int end, int norm) {
    if (m <= 1) return 1;
    if (m == 2) return n <= 9472 && (end == FEW_ROTARY || k < 4096);
    if (m <= 4) return end == FEW_ROTARY ? n <= 6144 : end == FEW_GATED ? n <= 8192 && k <= 1024 : n <= 8192 && k <= 128;
    return end != FEW_PLAIN && norm && n <= 1024 && k <= 512;
}

// gemm_simt for few rows with the work that `fusion` asks for; out is [m][n], of a gated unit [m][n / 2].
FR_EXPORT int gemm_simt_few(const float* a, const float* w, float* out, const void* bias, int bias_dtype, const float* residual, int m, int n,
                            int k, int lda, int ldw, int ldo, const GemmFewFusion* fusion, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return FR_OK;
    const GemmFewFusion& f = *fusion;
    if (!gemm_simt_few_supports(a, w, m, n, k, lda, ldw)) FR_REFUSE("gemm_simt (few rows): %d x %d x %d, strides %d and %d", m, n, k, lda, ldw);
    if (f.nq > 0 && (f.act || residual != nullptr || f.nkv <= 0 || f.hd <= 0 || (f.hd & 1) || (f.rot & 1) || f.rot < 0 || f.rot > f.hd ||
                     n != (f.nq + 2 * f.nkv) * f.hd || f.row_seq == nullptr || f.row_pos == nullptr || (f.denom != nullptr && f.rot == 0)))
        FR_REFUSE("gemm_simt (few rows): %d + 2 x %d heads of %d with %d rotated in %d columns", f.nq, f.nkv, f.hd, f.rot, n);
    if (f.act && ((n & 1) || residual != nullptr)) FR_REFUSE("gemm_simt (few rows): a gated unit of %d columns", n);
    const F32Args p{a, w, out, FrVec{bias, bias_dtype}, residual, m, n, k, lda, ldw, ldo, 1, 0, f.fixed_weights};
    const bool wide = n >= 2368;                               // as many pairs per warp as keep the SMs' loads in flight
    if (m == 1) return wide ? launch_few_fused<1, 2>(p, f, stream) : launch_few_fused<1, 1>(p, f, stream);
    if (m == 2) return wide ? launch_few_fused<2, 2>(p, f, stream) : launch_few_fused<2, 1>(p, f, stream);
    if (m <= 4) return wide ? launch_few_fused<4, 2>(p, f, stream) : launch_few_fused<4, 1>(p, f, stream);
    return wide ? launch_few_fused<8, 2>(p, f, stream) : launch_few_fused<8, 1>(p, f, stream);
}
