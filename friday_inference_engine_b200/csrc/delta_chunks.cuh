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
// (the blocked form of the rule by its triangular system: Yang et al., "Parallelizing linear transformers with the delta rule over
// sequence length", 2024).  The walk along a sequence is then three small products per chunk instead of sixteen tokens' chains of sums.
// Ratios of decays are running products, never quotients or differences of logarithms.
//
// Two kernels.  The first prepares every chunk of every head (A, B, the triangular solution by forward substitution, a thread per
// channel), all of them at a time, in 64 bits: its results round once, when they are stored.  The second walks the chunks: a block owns
// one head of one sequence and 64 value channels; four warps fetch the prepared operands two chunks ahead, four warps, 16 value channels
// each, walk.  W S0 and S0^T (Gamma q) run on the tensor cores (mma.sync.m16n8k16): a warp keeps its channels' transposed state, fp32,
// in the layout of the instruction's accumulators, which is also that of its first operand.  Their operands are three bf16 numbers (hi +
// mid + lo: all 24 bits of magnitudes above 2^-110, fewer below) and a product the six partial products that reach 2^-18 of it; hi hi has an
// accumulator of its own, whose sums over 16 key channels are added in fp32 registers.  What goes into a result as it is, the sum over B
// and the state's decay and sum, are fp32 multiply-adds, which round: on the tensor cores, whose accumulators drop bits, the state's
// error was up to 1.2 times that of the walk token by token.
//
// Errors against 64 bits, in units of those token by token (norms, three sequences of up to 400 tokens, decays of exp(-0.03) to exp(-2) a
// token, keys with something or nothing in common): outputs 0.69 to 0.97, states 0.91 to 1.00 (nearly parallel keys 1.02).  Measured on B200, heads of 128, us token by token and so, with
// a decay per head and per channel: 16 heads, 8 prompts of 64 to 512 tokens 300 -> 202 and 618 -> 241, one of 2,048 552 -> 480 and 913 -> 516;
// 32 heads, 16 of 300 857 -> 880 and 2,990 -> 1,032 (with both products of the state on the tensor cores and the preparation in fp32: 155 and 181, 365 and
// 387, 640 and 737).
#pragma once
#include "mma_sync.cuh"

namespace {

constexpr int CT = 16;               // tokens per chunk
constexpr int CD = 128;              // key channels (zeros beyond dk)
constexpr int CV = 64;               // value channels per block
constexpr int CLD = CD + 8;          // bf16 numbers per row: eight rows' 16-byte pieces lie in different banks
constexpr int WALK_THREADS = 128, FETCH_THREADS = 128, PREP_THREADS = 256;
constexpr int CHUNK_STAGES = 3;      // prepared chunks in a walking block's shared memory

struct ChunkOperands {               // a prepared chunk of one head
    bf16 w[3][CT][CLD], q[3][CT][CLD];
    float k[CT][CD];                 // Gamma_16 / Gamma_s k_s
    float b[CT][CT];                 // B_ts at [s][t]
    float gamma[CD];
};
typedef float ChunkValues[CT][CV + 4];                       // U0 of 64 value channels
struct PrepShared {
    ChunkOperands ops;
    double q[CT][CD], k[CT][CD];     // its rows as they come
    double g[CT][CD];                // decays (one per token in the first row where a head has one)
    double a[CT][CT];
    double beta[CT];
};
struct WalkShared {
    ChunkOperands ops[CHUNK_STAGES];
    ChunkValues u0[CHUNK_STAGES];
};
static_assert(sizeof(ChunkOperands) % 16 == 0 && sizeof(ChunkValues) % 16 == 0, "copied in 16-byte pieces");

struct ChunkArgs {
    ScanArgs s;
    ChunkOperands* ops;              // [slots][heads of this call]
    ChunkValues* u0;                 // [slots][heads of this call][value_blocks]
    int head0, heads, value_blocks;  // the heads of this call
};
// Sequences' chunks lie one after another: a sequence's first row is no multiple of 16, so each may leave one slot empty.
__device__ __forceinline__ long long chunk_slot(int r0, int seq, int c) { return r0 / CT + seq + c; }

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
// Tiles' products a b, b of tile i in b[i / 2], columns of place i % 2: large += hi hi; small += the five others that count.  Tile after
// tile, so that an instruction does not wait for the one before it.
template <int TILES>
__device__ __forceinline__ void mma_split(float (&large)[TILES][4], float (&small)[TILES][4], const uint32_t (&a)[3][4], const uint32_t (&b)[TILES / 2][3][4]) {
    constexpr int PA[6] = {0, 0, 2, 1, 0, 1}, PB[6] = {0, 2, 0, 1, 1, 0};
#pragma unroll
    for (int x = 0; x < 6; ++x)
#pragma unroll
        for (int i = 0; i < TILES; ++i) {
            const uint32_t(&bt)[4] = b[i / 2][PB[x]];
            mma_16816(x == 0 ? large[i] : small[i], a[PA[x]], bt[2 * (i % 2)], bt[2 * (i % 2) + 1]);
        }
}
template <int N>
__device__ __forceinline__ void clear(float (&v)[N][4]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[i][e] = 0.f;
}
template <int N>
__device__ __forceinline__ void add_to(float (&sum)[N][4], const float (&v)[N][4]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[i][e] += v[i][e];
}
typedef unsigned long long Pair2;    // two floats
__device__ __forceinline__ Pair2 pair_of(float lo, float hi) { return (Pair2)__float_as_uint(lo) | (Pair2)__float_as_uint(hi) << 32; }
__device__ __forceinline__ void fma_pair2(Pair2& acc, Pair2 x, Pair2 y) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y)); }
__device__ __forceinline__ void walk_bar_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(WALK_THREADS + FETCH_THREADS) : "memory"); }
__device__ __forceinline__ void walk_bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(WALK_THREADS + FETCH_THREADS) : "memory"); }
constexpr int BAR_FULL = 1, BAR_EMPTY = 1 + CHUNK_STAGES;     // one of each per stage

template <typename TR, bool PER_CHANNEL>
__global__ void __launch_bounds__(PREP_THREADS, 2) delta_prepare_chunks_kernel(const ChunkArgs args) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    PrepShared& sm = *(PrepShared*)chunk_smem;
    const ScanArgs& p = args.s;
    const int c = blockIdx.x, head = args.head0 + blockIdx.y, seq = blockIdx.z;
    const int who = threadIdx.x, warp = who >> 5, lane = who & 31;
    const int r0 = p.seq_start[seq], n = p.seq_qlen[seq];
    fr_pdl_wait();
    fr_pdl_launch();
    const int t0 = c * CT, nt = min(CT, n - t0);
    if (nt <= 0 || p.row_seq[r0] < 0) return;
    const int group = head / (p.heads / p.qk_heads);
    const int qk = p.qk_heads * p.dk, channels = 2 * qk + p.heads * p.dv;
    const size_t at = (size_t)chunk_slot(r0, seq, c) * args.heads + blockIdx.y;
    const FrVec alog{p.a_log, p.vec_dtype}, dtb{p.dt_bias, p.vec_dtype};
    const float rate = expf(alog.at(head));
    ChunkOperands& o = sm.ops;
    // rows (a token beyond the sequence: no decay, no key, no correction)
#pragma unroll
    for (int it = 0; it < CT * CD / 4 / PREP_THREADS; ++it) {
        const int idx = who + it * PREP_THREADS, t = idx / (CD / 4), i = idx % (CD / 4) * 4;
        float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f), k4 = q4;
        if (t < nt && i < p.dk) {
            const float* row = p.qkv + (size_t)(r0 + t0 + t) * channels + group * p.dk + i;
            q4 = *(const float4*)row;
            k4 = *(const float4*)(row + qk);
        }
        *(double2*)&sm.q[t][i] = make_double2(q4.x, q4.y);
        *(double2*)&sm.q[t][i + 2] = make_double2(q4.z, q4.w);
        *(double2*)&sm.k[t][i] = make_double2(k4.x, k4.y);
        *(double2*)&sm.k[t][i + 2] = make_double2(k4.z, k4.w);
    }
    if (PER_CHANNEL) {
#pragma unroll
        for (int it = 0; it < CT * CD / PREP_THREADS; ++it) {
            const int idx = who + it * PREP_THREADS, t = idx / CD, i = idx % CD;
            sm.g[t][i] = t < nt && i < p.dk ? expf(-rate * softplus_f(raw_at<TR>(p.a_raw, (size_t)(r0 + t0 + t) * p.ld_a + head * p.dk + i) + dtb.at(head * p.dk + i))) : 1.f;
        }
    } else if (who < CT) {
        sm.g[0][who] = who < nt ? expf(-rate * softplus_f(raw_at<TR>(p.a_raw, (size_t)(r0 + t0 + who) * p.ld_a + head) + dtb.at(head))) : 1.f;
    }
    if (who < CT) sm.beta[who] = who < nt ? 1.0f / (1.0f + expf(-raw_at<TR>(p.b_raw, (size_t)(r0 + t0 + who) * p.ld_b + head))) : 0.f;
    __syncthreads();
    // A and B, a column s per warp and turn: the key of token s as the tokens after it see it
#pragma unroll 1
    for (int turn = 0; turn < 2; ++turn) {
        const int s = turn == 0 ? warp : CT - 1 - warp;
        double val[32];                                       // A_ts of t = 0 .. 15, then B_ts
        double2 x = *(const double2*)&sm.k[s][2 * lane], y = *(const double2*)&sm.k[s][64 + 2 * lane];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            val[t] = val[CT + t] = 0.0;
            if (t >= s) {
                const double2 q0 = *(const double2*)&sm.q[t][2 * lane], q1 = *(const double2*)&sm.q[t][64 + 2 * lane];
                if (t > s) {
                    const double2 k0 = *(const double2*)&sm.k[t][2 * lane], k1 = *(const double2*)&sm.k[t][64 + 2 * lane];
                    if (PER_CHANNEL) {
                        const double2 g0 = *(const double2*)&sm.g[t][2 * lane], g1 = *(const double2*)&sm.g[t][64 + 2 * lane];
                        x.x *= g0.x; x.y *= g0.y; y.x *= g1.x; y.y *= g1.y;
                    } else {
                        const double g = sm.g[0][t];
                        x.x *= g; x.y *= g; y.x *= g; y.y *= g;
                    }
                    val[t] = fma(x.x, k0.x, x.y * k0.y) + fma(y.x, k1.x, y.y * k1.y);
                }
                val[CT + t] = fma(x.x, q0.x, x.y * q0.y) + fma(y.x, q1.x, y.y * q1.y);
            }
        }
        // every value summed over the lanes; lane l ends with the l-th
#pragma unroll
        for (int half = 16; half > 0; half >>= 1) {
            const bool upper = (lane & half) != 0;
#pragma unroll
            for (int v = 0; v < half; ++v) {
                const double give = upper ? val[v] : val[v + half], keep = upper ? val[v + half] : val[v];
                val[v] = keep + __shfl_xor_sync(0xffffffffu, give, half);
            }
        }
        const int t = lane & (CT - 1);
        if (lane < CT) sm.a[t][s] = val[0];
        else o.b[s][t] = (float)val[0];
    }
    __syncthreads();
    // the triangular solutions, a thread per channel
    auto solve = [&](double (&x)[CT]) {                       // x: right hand sides without beta, then the solutions
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            double r0s = 0.0, r1s = 0.0;
#pragma unroll
            for (int s = 0; s < t; s += 2) {
                const double2 row = *(const double2*)&sm.a[t][s];
                r0s = fma(row.x, x[s], r0s);
                if (s + 1 < t) r1s = fma(row.y, x[s + 1], r1s);
            }
            x[t] = sm.beta[t] * (x[t] - (r0s + r1s));
        }
    };
    double x[CT];
    if (who < CD) {
        double gam = 1.0;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            gam *= PER_CHANNEL ? sm.g[t][who] : sm.g[0][t];
            x[t] = gam * sm.k[t][who];
            split3((float)(gam * sm.q[t][who]), o.q[0][t][who], o.q[1][t][who], o.q[2][t][who]);
        }
        o.gamma[who] = (float)gam;
        solve(x);
#pragma unroll
        for (int t = 0; t < CT; ++t) split3((float)x[t], o.w[0][t][who], o.w[1][t][who], o.w[2][t][who]);
    } else {
        const int i = who - CD;
        double left = 1.0;
#pragma unroll
        for (int t = CT - 1; t >= 0; --t) {
            o.k[t][i] = (float)(left * sm.k[t][i]);
            left *= PER_CHANNEL ? sm.g[t][i] : sm.g[0][t];
        }
        for (int j = i; j < args.value_blocks * CV; j += PREP_THREADS - CD) {
#pragma unroll
            for (int t = 0; t < CT; ++t)
                x[t] = t < nt && j < p.dv ? p.qkv[(size_t)(r0 + t0 + t) * channels + 2 * qk + head * p.dv + j] : 0.f;
            solve(x);
            float* u = &args.u0[at * args.value_blocks + j / CV][0][j % CV];
#pragma unroll
            for (int t = 0; t < CT; ++t) u[t * (CV + 4)] = (float)x[t];
        }
    }
    __syncthreads();
    uint4* dst = (uint4*)(args.ops + at);
    for (int i = who; i < (int)(sizeof(ChunkOperands) / 16); i += PREP_THREADS) dst[i] = ((const uint4*)&sm.ops)[i];
}

// the walking block's operands, two chunks ahead of the walk
__device__ __forceinline__ void fetch_chunks(const ChunkArgs& args, WalkShared& sm, int r0, int seq, int chunks) {
    const int who = threadIdx.x - WALK_THREADS;
    auto copy = [&](void* dst, const void* src, int bytes) {
        for (int i = who * 16; i < bytes; i += FETCH_THREADS * 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared((char*)dst + i)), "l"((const char*)src + i) : "memory");
    };
    constexpr int AHEAD = CHUNK_STAGES - 1;
    for (int c = 0; c < chunks + AHEAD; ++c) {
        if (c < chunks) {
            const int stage = c % CHUNK_STAGES;
            if (c >= CHUNK_STAGES) walk_bar_sync(BAR_EMPTY + stage);
            const size_t at = (size_t)chunk_slot(r0, seq, c) * args.heads + blockIdx.y;
            copy(&sm.ops[stage], args.ops + at, sizeof(ChunkOperands));
            copy(&sm.u0[stage], args.u0 + at * args.value_blocks + blockIdx.x, sizeof(ChunkValues));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (c >= AHEAD) {
            asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
            walk_bar_arrive(BAR_FULL + (c - AHEAD) % CHUNK_STAGES);
        }
    }
}

__device__ __forceinline__ void walk_chunks(const ScanArgs& p, WalkShared& sm, int r0, int n, int seq, int head, int col0) {
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
    for (int c = 0; c < chunks; ++c) {
        const int stage = c % CHUNK_STAGES;
        const ChunkOperands& o = sm.ops[stage];
        walk_bar_sync(BAR_FULL + stage);
        // W S0 (tiles 0 and 1: tokens 0-7 and 8-15) and (Gamma q) S0 (2 and 3)
        float sum[4][4], large[4][4], small[4][4];
        clear(sum);
        clear(small);
#pragma unroll
        for (int ks = 0; ks < CD / 16; ++ks) {
            uint32_t a[3][4], b[2][3][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float* v = s[2 * ks + (r >> 1)] + 2 * (r & 1);
                split3(v[0], v[1], a[0][r], a[1][r], a[2][r]);
            }
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) {
                ldsm4(b[0][pl], &o.w[pl][row_n][ks * 16 + at_n]);
                ldsm4(b[1][pl], &o.q[pl][row_n][ks * 16 + at_n]);
            }
            clear(large);
            mma_split<4>(large, small, a, b);
            add_to(sum, large);
        }
        add_to(sum, small);
        float u[2][4], out2[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                u[i][e] = sm.u0[stage][8 * i + 2 * t + (e & 1)][local + (e < 2 ? 0 : 8)] - sum[i][e];
                out2[i][e] = sum[2 + i][e];
            }
        // every token's correction of this lane's two columns
        float ul[CT], uh[CT];
#pragma unroll
        for (int src = 0; src < CT; ++src) {
            const int from = (lane & ~3) | ((src & 7) >> 1);
            ul[src] = __shfl_sync(0xffffffffu, u[src >> 3][src & 1], from);
            uh[src] = __shfl_sync(0xffffffffu, u[src >> 3][2 + (src & 1)], from);
        }
        // (a token's correction reaches itself and those after it only, whatever its value is)
#pragma unroll
        for (int src = 0; src < CT; ++src)
#pragma unroll
            for (int i = src >> 3; i < 2; ++i) {
                const float2 w = *(const float2*)&o.b[src][8 * i + 2 * t];
                if (8 * i + 2 * t >= src) {
                    out2[i][0] = fmaf(w.x, ul[src], out2[i][0]);
                    out2[i][2] = fmaf(w.x, uh[src], out2[i][2]);
                }
                if (8 * i + 2 * t + 1 >= src) {
                    out2[i][1] = fmaf(w.y, ul[src], out2[i][1]);
                    out2[i][3] = fmaf(w.y, uh[src], out2[i][3]);
                }
            }
        float* out = p.out + (size_t)(r0 + c * CT) * ((size_t)p.heads * p.dv) + (size_t)head * p.dv;
        const int nt = min(CT, n - c * CT);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tok = 8 * i + 2 * t + (e & 1), col = e < 2 ? c_lo : c_hi;
                if (tok < nt && col < p.dv) out[(size_t)tok * p.heads * p.dv + col] = out2[i][e];
            }
        // two channels of a column per instruction
        Pair2 pl[CT], ph[CT];
#pragma unroll
        for (int src = 0; src < CT; ++src) {
            pl[src] = pair_of(ul[src], ul[src]);
            ph[src] = pair_of(uh[src], uh[src]);
        }
#pragma unroll
        for (int j0 = 0; j0 < CD / 8; j0 += 4) {              // four tiles of eight key channels at a time
            Pair2 lo[4], hi[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 gam = *(const float2*)&o.gamma[8 * (j0 + j) + 2 * t];
                float(&v)[4] = s[j0 + j];
                lo[j] = pair_of(gam.x * v[0], gam.y * v[1]);
                hi[j] = pair_of(gam.x * v[2], gam.y * v[3]);
            }
#pragma unroll
            for (int src = 0; src < CT; ++src)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const Pair2 k2 = *(const Pair2*)&o.k[src][8 * (j0 + j) + 2 * t];
                    fma_pair2(lo[j], k2, pl[src]);
                    fma_pair2(hi[j], k2, ph[src]);
                }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float(&v)[4] = s[j0 + j];
                v[0] = __uint_as_float((uint32_t)lo[j]); v[1] = __uint_as_float((uint32_t)(lo[j] >> 32));
                v[2] = __uint_as_float((uint32_t)hi[j]); v[3] = __uint_as_float((uint32_t)(hi[j] >> 32));
            }
        }
        if (c + CHUNK_STAGES < chunks) walk_bar_arrive(BAR_EMPTY + stage);
    }
#pragma unroll
    for (int j = 0; j < CD / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = 8 * j + 2 * t + (e & 1), col = e < 2 ? c_lo : c_hi;
            if (i < p.dk && col < p.dv) S[(size_t)i * p.dv + col] = s[j][e];
        }
}

// RANKED: blocks in order of their sequences' lengths, the longest first, so that an SM's second block is a short one.  Taken where there are
// more blocks than SMs and sequences are shorter than three quarters of the longest on average (and at most 64 of them, many even out by
// themselves): 8 prompts of 64 to 512 tokens, 16 heads 177 us, in the order of the sequences 203; but 16 of 300 each,
// 32 heads, 696 and 661, since the compiler schedules the walk's instructions less well around it.
constexpr int WALK_RANKED = 64;
__device__ __forceinline__ int walked_sequence(const ScanArgs& p, int n_seqs, int rank) {
    __shared__ int lens[WALK_RANKED], found;
    const int i = threadIdx.x;
    if (i < n_seqs) lens[i] = p.seq_qlen[i];
    __syncthreads();
    if (i < n_seqs) {
        int before = 0;
        for (int j = 0; j < n_seqs; ++j) before += lens[j] > lens[i] || (lens[j] == lens[i] && j < i);
        if (before == rank) found = i;
    }
    __syncthreads();
    return found;
}

template <bool RANKED>
__global__ void __launch_bounds__(WALK_THREADS + FETCH_THREADS, 1) delta_walk_chunks_kernel(const ChunkArgs args, int n_seqs) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    WalkShared& sm = *(WalkShared*)chunk_smem;
    const ScanArgs& p = args.s;
    const int seq = RANKED ? walked_sequence(p, n_seqs, blockIdx.z) : blockIdx.z, head = args.head0 + blockIdx.y;
    const int r0 = p.seq_start[seq], n = p.seq_qlen[seq];
    fr_pdl_wait();
    fr_pdl_launch();
    if (n <= 0 || p.row_seq[r0] < 0) return;
    if (threadIdx.x < WALK_THREADS) walk_chunks(p, sm, r0, n, seq, head, blockIdx.x * CV);
    else fetch_chunks(args, sm, r0, seq, (n + CT - 1) / CT);
}

long long chunk_slots(int rows, int n_seqs) { return (long long)rows / CT + n_seqs + 1; }
long long chunk_head_bytes(int rows, int n_seqs, int dv) {                 // scratch of one head
    return chunk_slots(rows, n_seqs) * (long long)(sizeof(ChunkOperands) + (dv + CV - 1) / CV * sizeof(ChunkValues));
}
// Heads go in equal rounds of what this holds (0: not even one head fits).  Twice what 16 heads of 128 with 2,048 tokens take; half of it
// would cost them a second round.
constexpr long long CHUNK_SCRATCH = 128ll << 20;
int chunk_heads(int rows, int n_seqs, int heads, int dv) {
    const long long fit = CHUNK_SCRATCH / chunk_head_bytes(rows, n_seqs, dv);
    if (fit < 1) return 0;
    const long long rounds = (heads + fit - 1) / fit;
    return (int)((heads + rounds - 1) / rounds);
}

template <typename TR, bool PER_CHANNEL>
int launch_chunks(const ScanArgs& s, int rows, int n_seqs, int max_q_len, void* scratch, cudaStream_t stream) {
    static std::atomic<unsigned long long> configured{0};     // devices (as bits) on which the limits have been raised
    int device = 0;
    FR_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= 64) FR_REFUSE("delta chunks: device %d is outside the table of 64", device);
    if (!(configured.load(std::memory_order_acquire) & (1ull << device))) {
        FR_CUDA(cudaFuncSetAttribute(delta_prepare_chunks_kernel<TR, PER_CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PrepShared)));
        FR_CUDA(cudaFuncSetAttribute(delta_walk_chunks_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WalkShared)));
        FR_CUDA(cudaFuncSetAttribute(delta_walk_chunks_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WalkShared)));
        configured.fetch_or(1ull << device, std::memory_order_release);
    }
    const int sms = fr_sm_count() > 0 ? fr_sm_count() : 148, at_once = chunk_heads(rows, n_seqs, s.heads, s.dv), blocks = (s.dv + CV - 1) / CV;
    for (int h = 0; h < s.heads; h += at_once) {
        ChunkArgs a{s, (ChunkOperands*)scratch, nullptr, h, s.heads - h < at_once ? s.heads - h : at_once, blocks};
        a.u0 = (ChunkValues*)(a.ops + chunk_slots(rows, n_seqs) * a.heads);
        FR_CUDA(fr_launch(delta_prepare_chunks_kernel<TR, PER_CHANNEL>, dim3((max_q_len + CT - 1) / CT, a.heads, n_seqs), dim3(PREP_THREADS), sizeof(PrepShared), stream, a));
        FR_CHECK_LAUNCH("delta chunks (prepare)");
        const bool ranked = n_seqs > 1 && n_seqs <= WALK_RANKED && (long long)blocks * a.heads * n_seqs > sms && 4ll * rows < 3ll * max_q_len * n_seqs;
        FR_CUDA(fr_launch(ranked ? delta_walk_chunks_kernel<true> : delta_walk_chunks_kernel<false>, dim3(blocks, a.heads, n_seqs),
                          dim3(WALK_THREADS + FETCH_THREADS), sizeof(WalkShared), stream, a, n_seqs));
        FR_CHECK_LAUNCH("delta chunks (walk)");
    }
    return FR_OK;
}

}  // namespace
