// The gated delta rule of prompts in chunks of 16 tokens.
//
// With Gamma_t the product of the decays up to token t of its chunk (elementwise, per key channel or one number), S0 the state
// before the chunk, and  A_ts = sum_c k_s k_t Gamma_t / Gamma_s  (s < t),  B_ts the same with q_t (s <= t),  the corrections
// u_t of a chunk solve a triangular system that does not need the state,
//
//     u_t + beta_t sum_(s < t) A_ts u_s = beta_t (v_t - S0^T (Gamma_t k_t))
//
// so that, with W and U0 its solutions for the right hand sides beta_t Gamma_t k_t and beta_t v_t,
//
//     U = U0 - W S0,    o_t = S0^T (Gamma_t q_t) + sum_(s <= t) B_ts u_s,    S = Gamma_16 S0 + sum_s (Gamma_16 / Gamma_s k_s) u_s^T.
//
// The walk along a sequence is then three small products per chunk instead of sixteen tokens' chains of sums.  Ratios of decays
// are running products, never quotients or differences of logarithms.
//
// A block owns one head of one sequence and 64 value channels.  Eight warps prepare a chunk (A, B, the triangular solution by
// forward substitution, a thread per channel; fp32) while four warps, 16 value channels each, walk the chunk before it on the
// tensor cores (mma.sync.m16n8k16): a warp keeps its channels' transposed state, fp32, in the layout of the instruction's
// accumulators, which is also that of its first operand, so that nothing but the prepared operands passes through shared memory.
// Every operand is three bf16 numbers (hi + mid + lo, all 24 bits) and a product the six partial products that reach
// 2^-18 of it; hi hi has an accumulator of its own, the state's decay and sum are fp32 multiply-adds, so that the errors stay
// those of fp32 sums.
#pragma once
#include "mma_sync.cuh"

namespace {

constexpr int CT = 16;               // tokens per chunk
constexpr int CD = 128;              // key channels (zeros beyond dk)
constexpr int CV = 64;               // value channels per block
constexpr int CLD = CD + 8;          // bf16 numbers per row: eight rows' 16-byte pieces lie in different banks
constexpr int CHAIN_THREADS = 128, PREP_THREADS = 256, CHUNK_THREADS = CHAIN_THREADS + PREP_THREADS;

struct ChunkOperands {               // a prepared chunk
    bf16 w[3][CT][CLD], q[3][CT][CLD], k[3][CT][CLD];
    bf16 b[3][CT][CT + 8];
    float u0[CT][CV + 4];
    float gamma[CD];
};
struct ChunkRaw {                    // its rows as they come
    float q[CT][CD], k[CT][CD], v[CT][CV];
};
struct ChunkShared {
    ChunkOperands ops[2];
    ChunkRaw raw[2];
    float g[CT][CD];                 // decays
    float a[CT][CT];
    float beta[CT];
};

__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack2(x, y);
    x -= __uint_as_float(hi << 16);
    y -= __uint_as_float(hi & 0xffff0000u);
    mid = pack2(x, y);
    x -= __uint_as_float(mid << 16);
    y -= __uint_as_float(mid & 0xffff0000u);
    lo = pack2(x, y);
}
__device__ __forceinline__ void split3(float x, bf16& hi, bf16& mid, bf16& lo) {
    hi = __float2bfloat16_rn(x);
    x -= __bfloat162float(hi);
    mid = __float2bfloat16_rn(x);
    x -= __bfloat162float(mid);
    lo = __float2bfloat16_rn(x);
}
// large += a_hi b_hi; small += the five others that count
__device__ __forceinline__ void mma_split(float (&large)[4], float (&small)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int tile) {
    mma_16816(large, a[0], b[0][2 * tile], b[0][2 * tile + 1]);
    mma_16816(small, a[0], b[2][2 * tile], b[2][2 * tile + 1]);
    mma_16816(small, a[2], b[0][2 * tile], b[0][2 * tile + 1]);
    mma_16816(small, a[1], b[1][2 * tile], b[1][2 * tile + 1]);
    mma_16816(small, a[0], b[1][2 * tile], b[1][2 * tile + 1]);
    mma_16816(small, a[1], b[0][2 * tile], b[0][2 * tile + 1]);
}
template <int ID, int THREADS>
__device__ __forceinline__ void named_sync() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory"); }
__device__ __forceinline__ void chunk_bar_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(CHUNK_THREADS) : "memory"); }
__device__ __forceinline__ void chunk_bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(CHUNK_THREADS) : "memory"); }
constexpr int BAR_PREP = 1, BAR_FULL = 2, BAR_EMPTY = 4;      // full and empty: one per buffer

template <typename TR, bool PER_CHANNEL>
__device__ __forceinline__ void prepare_chunks(const ScanArgs& p, ChunkShared& sm, int r0, int n, int head, int col0) {
    const int who = threadIdx.x - CHAIN_THREADS, warp = who >> 5, lane = who & 31;
    const int group = head / (p.heads / p.qk_heads);
    const int qk = p.qk_heads * p.dk, channels = 2 * qk + p.heads * p.dv;
    const FrVec alog{p.a_log, p.vec_dtype}, dtb{p.dt_bias, p.vec_dtype};
    const float rate = expf(alog.at(head));
    const int chunks = (n + CT - 1) / CT;
    constexpr int GZ = PER_CHANNEL ? CT * CD / PREP_THREADS : 1;
    float gz[GZ], zb = 0.f;
    // rows of chunk c: q, k, v into shared memory, raw decays and betas into registers
    auto fetch = [&](int c) {
        const int t0 = c * CT, nt = min(CT, n - t0);
        ChunkRaw& raw = sm.raw[c & 1];
        auto copy = [&](float* dst, const float* src, bool there) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(there ? src : p.qkv), "r"(there ? 16 : 0)
                         : "memory");
        };
#pragma unroll
        for (int it = 0; it < CT * CD / 4 / PREP_THREADS; ++it) {
            const int idx = who + it * PREP_THREADS, t = idx / (CD / 4), i = idx % (CD / 4) * 4;
            const bool there = t < nt && i < p.dk;
            const float* row = p.qkv + (size_t)(r0 + t0 + (there ? t : 0)) * channels + group * p.dk + i;
            copy(&raw.q[t][i], row, there);
            copy(&raw.k[t][i], row + qk, there);
        }
        static_assert(CT * CV / 4 == PREP_THREADS, "a piece of the values per thread");
        const int t = who / (CV / 4), j = who % (CV / 4) * 4;
        const bool there = t < nt && col0 + j < p.dv;
        copy(&raw.v[t][j], p.qkv + (size_t)(r0 + t0 + (there ? t : 0)) * channels + 2 * qk + head * p.dv + col0 + (there ? j : 0), there);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (PER_CHANNEL) {
#pragma unroll
            for (int it = 0; it < GZ; ++it) {
                const int idx = who + it * PREP_THREADS, tt = idx / CD, i = idx % CD;
                gz[it] = tt < nt && i < p.dk ? raw_at<TR>(p.a_raw, (size_t)(r0 + t0 + tt) * p.ld_a + head * p.dk + i) : 0.f;
            }
        } else {
            gz[0] = who < nt ? raw_at<TR>(p.a_raw, (size_t)(r0 + t0 + who) * p.ld_a + head) : 0.f;
        }
        zb = who < nt ? raw_at<TR>(p.b_raw, (size_t)(r0 + t0 + who) * p.ld_b + head) : 0.f;
    };
    fetch(0);
    for (int c = 0; c < chunks; ++c) {
        const int nt = min(CT, n - c * CT), buf = c & 1;
        const ChunkRaw& raw = sm.raw[buf];
        ChunkOperands& o = sm.ops[buf];
        // decays and betas (a token beyond the sequence: no decay, no key, no correction)
        if (PER_CHANNEL) {
#pragma unroll
            for (int it = 0; it < GZ; ++it) {
                const int idx = who + it * PREP_THREADS, t = idx / CD, i = idx % CD;
                sm.g[t][i] = t < nt && i < p.dk ? expf(-rate * softplus_f(gz[it] + dtb.at(head * p.dk + i))) : 1.f;
            }
        } else if (who < CT) {
            sm.g[0][who] = who < nt ? expf(-rate * softplus_f(gz[0] + dtb.at(head))) : 1.f;
        }
        if (who < CT) sm.beta[who] = who < nt ? 1.0f / (1.0f + expf(-zb)) : 0.f;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        named_sync<BAR_PREP, PREP_THREADS>();
        if (c >= 2) chunk_bar_sync(BAR_EMPTY + buf);
        if (c + 1 < chunks) fetch(c + 1);                     // (nobody reads that buffer any more: the barrier above)
        // A and B, a column s per warp and turn: the key of token s as the tokens after it see it
#pragma unroll
        for (int turn = 0; turn < 2; ++turn) {
            const int s = turn == 0 ? warp : CT - 1 - warp;
            float val[32];                                    // A_ts of t = 0 .. 15, then B_ts
            float4 x = *(const float4*)&raw.k[s][4 * lane];
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                val[t] = val[CT + t] = 0.f;
                if (t >= s) {
                    const float4 qt = *(const float4*)&raw.q[t][4 * lane];
                    if (t > s) {
                        const float4 kt = *(const float4*)&raw.k[t][4 * lane];
                        if (PER_CHANNEL) {
                            const float4 g = *(const float4*)&sm.g[t][4 * lane];
                            x.x *= g.x; x.y *= g.y; x.z *= g.z; x.w *= g.w;
                        } else {
                            const float g = sm.g[0][t];
                            x.x *= g; x.y *= g; x.z *= g; x.w *= g;
                        }
                        val[t] = fmaf(x.x, kt.x, x.y * kt.y) + fmaf(x.z, kt.z, x.w * kt.w);
                    }
                    val[CT + t] = fmaf(x.x, qt.x, x.y * qt.y) + fmaf(x.z, qt.z, x.w * qt.w);
                }
            }
            // every value summed over the lanes; lane l ends with the l-th
#pragma unroll
            for (int half = 16; half > 0; half >>= 1) {
                const bool upper = (lane & half) != 0;
#pragma unroll
                for (int v = 0; v < half; ++v) {
                    const float give = upper ? val[v] : val[v + half], keep = upper ? val[v + half] : val[v];
                    val[v] = keep + __shfl_xor_sync(0xffffffffu, give, half);
                }
            }
            const int t = lane & (CT - 1);
            if (lane < CT) sm.a[t][s] = val[0];
            else split3(val[0], o.b[0][t][s], o.b[1][t][s], o.b[2][t][s]);
        }
        named_sync<BAR_PREP, PREP_THREADS>();
        // the triangular solutions, a thread per channel
        auto solve = [&](float (&x)[CT]) {                    // x: right hand sides without beta, then the solutions
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                float r0s = 0.f, r1s = 0.f, r2s = 0.f, r3s = 0.f;
#pragma unroll
                for (int s = 0; s < t; s += 4) {
                    const float4 at = *(const float4*)&sm.a[t][s];
                    r0s = fmaf(at.x, x[s], r0s);
                    if (s + 1 < t) r1s = fmaf(at.y, x[s + 1], r1s);
                    if (s + 2 < t) r2s = fmaf(at.z, x[s + 2], r2s);
                    if (s + 3 < t) r3s = fmaf(at.w, x[s + 3], r3s);
                }
                x[t] = sm.beta[t] * (x[t] - ((r0s + r1s) + (r2s + r3s)));
            }
        };
        float x[CT];
        if (who < CD) {
            float gam = 1.f;
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                gam *= PER_CHANNEL ? sm.g[t][who] : sm.g[0][t];
                x[t] = gam * raw.k[t][who];
                split3(gam * raw.q[t][who], o.q[0][t][who], o.q[1][t][who], o.q[2][t][who]);
            }
            o.gamma[who] = gam;
            solve(x);
#pragma unroll
            for (int t = 0; t < CT; ++t) split3(x[t], o.w[0][t][who], o.w[1][t][who], o.w[2][t][who]);
        } else {
            const int i = who - CD;
            float left = 1.f;
#pragma unroll
            for (int t = CT - 1; t >= 0; --t) {
                split3(left * raw.k[t][i], o.k[0][t][i], o.k[1][t][i], o.k[2][t][i]);
                left *= PER_CHANNEL ? sm.g[t][i] : sm.g[0][t];
            }
            if (i < CV) {
#pragma unroll
                for (int t = 0; t < CT; ++t) x[t] = raw.v[t][i];
                solve(x);
#pragma unroll
                for (int t = 0; t < CT; ++t) o.u0[t][i] = x[t];
            }
        }
        chunk_bar_arrive(BAR_FULL + buf);
        if (c + 1 < chunks) named_sync<BAR_PREP, PREP_THREADS>();      // decays, A and rows may be written again
    }
}

__device__ __forceinline__ void walk_chunks(const ScanArgs& p, ChunkShared& sm, int r0, int n, int seq, int head, int col0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int c_lo = col0 + warp * 16 + g, c_hi = c_lo + 8, local = warp * 16 + g;
    const int chunks = (n + CT - 1) / CT;
    float* S = p.state + (size_t)p.seq_slots[seq] * p.state_stride + p.s_off + (size_t)head * p.dk * p.dv;
    float s[CD / 8][4];                                       // channels 8 j + 2 t, + 1 of columns c_lo and c_hi
#pragma unroll
    for (int j = 0; j < CD / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = 8 * j + 2 * t + (e & 1), col = e < 2 ? c_lo : c_hi;
            s[j][e] = i < p.dk && col < p.dv ? S[(size_t)i * p.dv + col] : 0.f;
        }
    const int mi = lane >> 3, row_n = (mi >> 1) * 8 + (lane & 7), at_n = (mi & 1) * 8;       // ldmatrix: [n][k] tiles
    const int row_t = (mi & 1) * 8 + (lane & 7), at_t = (mi >> 1) * 8;                       // transposed: [k][n] tiles
    for (int c = 0; c < chunks; ++c) {
        const int buf = c & 1;
        const ChunkOperands& o = sm.ops[buf];
        chunk_bar_sync(BAR_FULL + buf);
        float ul[2][4] = {}, us[2][4] = {}, ol[2][4] = {}, os[2][4] = {};     // W S0 and (Gamma q) S0, two tiles of 8 tokens each
#pragma unroll
        for (int ks = 0; ks < CD / 16; ++ks) {
            uint32_t a[3][4], b[3][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float* v = s[2 * ks + (r >> 1)] + 2 * (r & 1);
                split3(v[0], v[1], a[0][r], a[1][r], a[2][r]);
            }
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) ldsm4(b[pl], &o.w[pl][row_n][ks * 16 + at_n]);
            mma_split(ul[0], us[0], a, b, 0);
            mma_split(ul[1], us[1], a, b, 1);
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) ldsm4(b[pl], &o.q[pl][row_n][ks * 16 + at_n]);
            mma_split(ol[0], os[0], a, b, 0);
            mma_split(ol[1], os[1], a, b, 1);
        }
        float u[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) u[i][e] = o.u0[8 * i + 2 * t + (e & 1)][local + (e < 2 ? 0 : 8)] - (ul[i][e] + us[i][e]);
        uint32_t ua[3][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) split3(u[r >> 1][2 * (r & 1)], u[r >> 1][2 * (r & 1) + 1], ua[0][r], ua[1][r], ua[2][r]);
        float finite = 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) finite = fmaf(0.f, u[i][e], finite);
        if (!__any_sync(0xffffffffu, finite != finite)) {
            uint32_t b[3][4];
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) ldsm4(b[pl], &o.b[pl][row_n][at_n]);
            mma_split(ol[0], os[0], ua, b, 0);
            mma_split(ol[1], os[1], ua, b, 1);
        } else {
            // a correction that is not finite reaches its own token and those after it only: no product with a zero of B
#pragma unroll
            for (int src = 0; src < CT; ++src) {
                const int from = (lane & ~3) | ((src & 7) >> 1);
                const float lo = __shfl_sync(0xffffffffu, u[src >> 3][src & 1], from), hi = __shfl_sync(0xffffffffu, u[src >> 3][2 + (src & 1)], from);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int to = 8 * i + 2 * t + e;
                        if (to < src) continue;
                        const float w = __bfloat162float(o.b[0][to][src]) + (__bfloat162float(o.b[1][to][src]) + __bfloat162float(o.b[2][to][src]));
                        ol[i][e] = fmaf(w, lo, ol[i][e]);
                        ol[i][2 + e] = fmaf(w, hi, ol[i][2 + e]);
                    }
            }
        }
        float* out = p.out + (size_t)(r0 + c * CT) * ((size_t)p.heads * p.dv) + (size_t)head * p.dv;
        const int nt = min(CT, n - c * CT);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tok = 8 * i + 2 * t + (e & 1), col = e < 2 ? c_lo : c_hi;
                if (tok < nt && col < p.dv) out[(size_t)tok * p.heads * p.dv + col] = ol[i][e] + os[i][e];
            }
#pragma unroll
        for (int jt = 0; jt < CD / 16; ++jt) {
            uint32_t b[3][4];
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) ldsm4t(b[pl], &o.k[pl][row_t][jt * 16 + at_t]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int j = 2 * jt + i;
                float dl[4] = {}, ds[4] = {};
                mma_split(dl, ds, ua, b, i);
                const float2 gam = *(const float2*)&o.gamma[8 * j + 2 * t];
                s[j][0] = fmaf(gam.x, s[j][0], dl[0] + ds[0]);
                s[j][1] = fmaf(gam.y, s[j][1], dl[1] + ds[1]);
                s[j][2] = fmaf(gam.x, s[j][2], dl[2] + ds[2]);
                s[j][3] = fmaf(gam.y, s[j][3], dl[3] + ds[3]);
            }
        }
        if (c + 2 < chunks) chunk_bar_arrive(BAR_EMPTY + buf);
    }
#pragma unroll
    for (int j = 0; j < CD / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = 8 * j + 2 * t + (e & 1), col = e < 2 ? c_lo : c_hi;
            if (i < p.dk && col < p.dv) S[(size_t)i * p.dv + col] = s[j][e];
        }
}

template <typename TR, bool PER_CHANNEL>
__global__ void __launch_bounds__(CHUNK_THREADS, 1) delta_chunks_kernel(const ScanArgs p) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    ChunkShared& sm = *(ChunkShared*)chunk_smem;
    const int seq = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * CV;
    const int r0 = p.seq_start[seq], n = p.seq_qlen[seq];
    fr_pdl_wait();
    fr_pdl_launch();
    if (n <= 0 || p.row_seq[r0] < 0) return;
    if (threadIdx.x < CHAIN_THREADS) walk_chunks(p, sm, r0, n, seq, head, col0);
    else prepare_chunks<TR, PER_CHANNEL>(p, sm, r0, n, head, col0);
}

template <typename TR, bool PER_CHANNEL>
int launch_chunks(const ScanArgs& p, int n_seqs, cudaStream_t stream) {
    static std::atomic<unsigned long long> configured{0};     // devices (as bits) on which the limit has been raised
    int device = 0;
    FR_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= 64) FR_REFUSE("delta chunks: device %d is outside the table of 64", device);
    if (!(configured.load(std::memory_order_acquire) & (1ull << device))) {
        FR_CUDA(cudaFuncSetAttribute(delta_chunks_kernel<TR, PER_CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChunkShared)));
        configured.fetch_or(1ull << device, std::memory_order_release);
    }
    FR_CUDA(fr_launch(delta_chunks_kernel<TR, PER_CHANNEL>, dim3(n_seqs, p.heads, (p.dv + CV - 1) / CV), dim3(CHUNK_THREADS), sizeof(ChunkShared), stream, p));
    FR_CHECK_LAUNCH("delta chunks");
    return FR_OK;
}

}  // namespace
