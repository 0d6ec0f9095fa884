// The 32-bit product of many rows on the tensor cores.
//
// Every fp32 operand is the sum of three bf16 numbers, x = hi + mid + lo, each the rounding of what the ones before it
// leave: 8 + 8 + 8 significant bits, so none of the 24 is lost (the split of a matrix into parts whose products are exact is Ozaki, Ogita, Oishi and
// Rump's, "Error-free transformations of matrix multiplication", 2012).  A product is the sum of the six partial products that
// reach 2^-18 of it (hi hi, hi mid, mid hi, hi lo, mid mid, lo hi; what is left out is below 2^-25), which the tensor
// core forms exactly and adds in fp32.  Its accumulators drop the bits of an addend below the sum's last place instead of
// rounding, an error that grows with the number of additions.  So hi hi has an accumulator of its own, which sums 128 of k
// at a time (eight additions); these parts are added in fp32 registers.  The five small products share another accumulator
// over all of k: its values, and with them what it drops, are 2^-8 of the others.
//
// Where all of a tile's weights in a block of k are bf16 numbers already (a bf16 checkpoint run in 32 bits: every block),
// their mid and lo are zero and the three products with them are not issued: the result is the same.
//
// A value that no sum of three bf16 numbers is (not finite, or so near the largest float that hi would round to infinity)
// marks its row; results of marked rows are computed by fp32 multiply-adds instead, so that infinities and
// NaN come out as they do everywhere else.  bf16 ends at 2^-133, so magnitudes below 2^-110 have fewer than 24 bits in three of them: rows of x
// that lie below 2^-63 as a whole are split times 2^64 and their results divided by it, weight rows of that kind (that are no bf16
// numbers) are marked.  What is left is a value below 2^-110 in a row that reaches 2^-63: off by 2^-134, 2^-71 of the row's largest.
//
// Weights lie on the M side (128 columns of the result per tile), rows of x on the N side.  x is split once by a kernel of
// its own into three planes in memory and comes by TMA.  Weights come by TMA as they are, 32 of k at a time; four converter
// warps split them and write the planes into TENSOR memory, from where the instruction takes its A operand: a split through
// shared memory would make its bandwidth the bound (each block of k would cross it five times instead of twice).  Eight
// warps add the parts; one lane each issues copies and instructions.  k is split over the CTAs of a cluster where there are
// few tiles; the parts are added in order of k through distributed shared memory.
//
// Measured on B200, us, this kernel (with the split of x) against the register tiles of gemm_simt.cu, weights that are bf16
// numbers (and that are not): 333 x 37888 x 3584 320 (450) against 1,896, 333 x 3584 x 18944 207 (264) against 1,064, 333 x 4608 x
// 3584 52 (63) against 256, 64 x 3584 x 3584 28 against 83, 24 x 37888 x 3584 157 against 207.  Relative error against 64 bits for
// normal values, both in turn: k = 256 1.2e-7 and 2.1e-7, 1,024 1.3e-7 and 1.6e-7, 3,584 1.5e-7 and 5.4e-7, 18,944 2.4e-7
// and 8.7e-7.
#pragma once
#include "tc_common.cuh"

#include <atomic>

namespace {

using namespace tc;

constexpr int SPLIT_BK = 32;                                   // of k per stage: 128 bytes of weights, 64 of each plane
constexpr int SPLIT_BN = 176;                                  // rows of x per tile at most: both accumulators and three stages of weights fill tensor memory
constexpr int SPLIT_GROUP = 4;                                 // blocks of k that the accumulator of hi hi sums at a time
constexpr int SPLIT_W_BYTES = TILE_P * SPLIT_BK * 4;
constexpr int SPLIT_W_STAGES = 5, SPLIT_A_STAGES = 3;
constexpr int SPLIT_X_STAGES = 10;                             // at most (of small tiles)
constexpr int SPLIT_A_COLS = 3 * SPLIT_BK / 2;                 // tensor-memory columns of a stage: two bf16 per column, three planes
constexpr int SPLIT_A0 = 2 * SPLIT_BN;
constexpr int SPLIT_TMEM = 512;
static_assert(SPLIT_A0 + SPLIT_A_STAGES * SPLIT_A_COLS <= SPLIT_TMEM, "accumulators and weights share tensor memory");
constexpr int SPLIT_THREADS = 14 * 32;                         // four warps split weights, eight add, one copies, one issues products
constexpr int SPLIT_STATIC_SMEM = 2048;                        // barriers and flags, which are not part of the dynamic memory
constexpr int SPLIT_MAX_SMEM = 227 * 1024 - SPLIT_STATIC_SMEM;
constexpr int SPLIT_FIXED_SMEM = 1024 + SPLIT_W_STAGES * SPLIT_W_BYTES;    // (1,024 for the alignment)

constexpr int SPLIT_BAD = 1, SPLIT_TINY = 2;
constexpr uint32_t SPLIT_LARGE_BITS = 0x60000000u;             // some of these are set in magnitudes from 2^-63 on, none in those below

struct SplitArgs {
    const float* x;
    const float* w;
    float* out;
    FrVec bias;
    const float* residual;
    const int* marked;               // [m] rows of x: SPLIT_BAD with a value that is no sum of three bf16, SPLIT_TINY times 2^64 in the planes
    int m, n, k, lda, ldw, ldo;
    int bn, tiles_q, x_stages, splits, kb_per, fixed_weights;
    int* status;
};

__device__ __forceinline__ uint64_t smem_desc_64(uint32_t addr) {     // K-major, rows of 64 bytes (64-byte swizzle), groups of 8 rows 512 bytes apart
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ void tc_mma_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void split_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {          // a in the low half
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *(const uint32_t*)&v;
}
// The roundings of two values, which keep what the rounding left.
__device__ __forceinline__ uint32_t take_bf16(float& a, float& b) {
    const uint32_t r = pack_bf16(a, b);
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
    return r;
}
// Two values into three pairs of bf16.  `bad` turns NaN and stays so if a value cannot be split (hi is infinite or NaN, so
// that something that is not finite is left).
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo, float& bad) {
    hi = take_bf16(a, b);
    mid = take_bf16(a, b);
    lo = pack_bf16(a, b);
    bad = fmaf(0.f, a + b, bad);
}

template <bool B>
struct Scaled {
    static constexpr bool value = B;
};

// x [m][k] into planes [3][m][kp] (kp: k up to a multiple of 8, zeros beyond k), a block per row.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ planes, int* __restrict__ marked, int m, int k, int kp, int lda) {
    __shared__ uint32_t s_seen;                                // SPLIT_BAD; 2: a magnitude from 2^-63 on; 4: one that is not zero
    if (threadIdx.x == 0) s_seen = 0u;
    __syncthreads();
    fr_pdl_wait();
    fr_pdl_launch();
    const int row = blockIdx.x;
    const float* src = x + (size_t)row * lda;
    const size_t plane = (size_t)m * kp;
    __nv_bfloat16* dst = planes + (size_t)row * kp;
    float bad = 0.f;
    uint32_t bits = 0u;
    auto split = [&](auto scaled) {
        for (int c = threadIdx.x * 8; c < kp; c += 256 * 8) {
            float4 a = *(const float4*)(src + c);
            float4 b = c + 4 < k ? *(const float4*)(src + c + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (decltype(scaled)::value) {
                a.x *= 0x1p64f; a.y *= 0x1p64f; a.z *= 0x1p64f; a.w *= 0x1p64f;
                b.x *= 0x1p64f; b.y *= 0x1p64f; b.z *= 0x1p64f; b.w *= 0x1p64f;
            } else {
                bits |= (__float_as_uint(a.x) | __float_as_uint(a.y)) | (__float_as_uint(a.z) | __float_as_uint(a.w));
                bits |= (__float_as_uint(b.x) | __float_as_uint(b.y)) | (__float_as_uint(b.z) | __float_as_uint(b.w));
            }
            uint4 hi, mid, lo;
            split_pair(a.x, a.y, hi.x, mid.x, lo.x, bad);
            split_pair(a.z, a.w, hi.y, mid.y, lo.y, bad);
            split_pair(b.x, b.y, hi.z, mid.z, lo.z, bad);
            split_pair(b.z, b.w, hi.w, mid.w, lo.w, bad);
            *(uint4*)(dst + c) = hi;
            *(uint4*)(dst + plane + c) = mid;
            *(uint4*)(dst + 2 * plane + c) = lo;
        }
    };
    split(Scaled<false>{});
    const uint32_t seen = __reduce_or_sync(0xffffffffu, (bad != bad ? SPLIT_BAD : 0u) | ((bits & SPLIT_LARGE_BITS) ? 2u : 0u) | ((bits & 0x7fffffffu) ? 4u : 0u));
    if ((threadIdx.x & 31) == 0 && seen != 0u) atomicOr(&s_seen, seen);
    __syncthreads();
    const bool tiny = s_seen == 4u;                            // (nothing so small is bad)
    if (tiny) split(Scaled<true>{});
    if (threadIdx.x == 0) marked[row] = tiny ? SPLIT_TINY : (s_seen & SPLIT_BAD);
}

// (rows lie in pieces of four; a part of 256 at a time, so that the error stays near that of the sums on the tensor cores)
__device__ __forceinline__ float split_plain_dot(const SplitArgs& p, int row, int col) {
    const float* a = p.x + (size_t)row * p.lda;
    const float* b = p.w + (size_t)col * p.ldw;
    float total = 0.f;
    for (int k0 = 0; k0 < p.k; k0 += 256) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        for (int i = k0; i < min(k0 + 256, p.k); i += 4) {
            const float4 u = *(const float4*)(a + i), v = *(const float4*)(b + i);
            s0 = fmaf(u.x, v.x, s0);
            s1 = fmaf(u.y, v.y, s1);
            s2 = fmaf(u.z, v.z, s2);
            s3 = fmaf(u.w, v.w, s3);
        }
        total += (s0 + s1) + (s2 + s3);
    }
    return total;
}

__global__ void __launch_bounds__(SPLIT_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const SplitArgs p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * SPLIT_W_STAGES + 2 * SPLIT_X_STAGES + 2 * SPLIT_A_STAGES + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_wide[SPLIT_A_STAGES][4];                  // a quarter of the stage's weights has mid or lo parts
    __shared__ float s_bad[TILE_P];                            // weight rows that cannot be split
    __shared__ float s_any;                                    // such a row, or a marked one of x, is among the tile's
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* x_ring = smem + SPLIT_W_STAGES * SPLIT_W_BYTES;
    const int bn = p.bn, XS = p.x_stages;
    const uint32_t x_bytes = 3u * bn * SPLIT_BK * 2;
    const uint32_t wfull = smem_u32(bars), wempty = wfull + 8 * SPLIT_W_STAGES;
    const uint32_t xfull = wempty + 8 * SPLIT_W_STAGES, xempty = xfull + 8 * SPLIT_X_STAGES;
    const uint32_t afull = xempty + 8 * SPLIT_X_STAGES, aempty = afull + 8 * SPLIT_A_STAGES;
    const uint32_t accf = aempty + 8 * SPLIT_A_STAGES, acce = accf + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / p.splits, split = blockIdx.x - tile * p.splits;
    const int q = tile % p.tiles_q, n0 = tile / p.tiles_q * TILE_P, m0 = q * bn;     // tiles that share weights run side by side
    const int kb0 = split * p.kb_per, kb1 = min((p.k + SPLIT_BK - 1) / SPLIT_BK, kb0 + p.kb_per);

    if (threadIdx.x == 0) {
        for (int s = 0; s < SPLIT_W_STAGES; ++s) {
            mbar_init(wfull + 8 * s, 1);
            mbar_init(wempty + 8 * s, 4);
        }
        for (int s = 0; s < XS; ++s) {
            mbar_init(xfull + 8 * s, 1);
            mbar_init(xempty + 8 * s, 1);
        }
        for (int s = 0; s < SPLIT_A_STAGES; ++s) {
            mbar_init(afull + 8 * s, 4);
            mbar_init(aempty + 8 * s, 1);
        }
        mbar_init(accf, 1);
        mbar_init(acce, 8);
        s_any = 0.f;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x < TILE_P) s_bad[threadIdx.x] = 0.f;
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)SPLIT_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (threadIdx.x == 0) fr_pdl_launch();

    if (warp < 4) {
        // ---- converters: a thread has one weight row
        const int quarter = warp & 3, row = quarter * 32 + lane, blocks = kb1 - kb0;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + SPLIT_A0;
        float bad4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t bits = 0u;                                    // all of the row's
        for (int i = 0; i < blocks; ++i) {
            const int ws = i % SPLIT_W_STAGES, as = i % SPLIT_A_STAGES;
            if (!mbar_wait(wfull + 8 * ws, (i / SPLIT_W_STAGES) & 1, p.status, 11)) break;
            float v[32];
            const uint8_t* src = smem + ws * SPLIT_W_BYTES + row * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 f = *(const float4*)(src + ((c ^ (row & 7)) << 4));
                v[4 * c] = f.x; v[4 * c + 1] = f.y; v[4 * c + 2] = f.z; v[4 * c + 3] = f.w;
            }
            uint32_t low[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int j = 0; j < 32; ++j) low[j & 3] |= __float_as_uint(v[j]);
            low[0] = (low[0] | low[1]) | (low[2] | low[3]);
            bits |= low[0];
            const bool wide = __any_sync(0xffffffffu, (low[0] & 0xffffu) != 0);
            if (lane == 0) mbar_arrive(wempty + 8 * ws);       // (the vote has seen every lane's loads)
            if (!mbar_wait(aempty + 8 * as, ((i / SPLIT_A_STAGES) & 1) ^ 1, p.status, 12)) break;
            tc_fence_after();
            const uint32_t dst = lane_base + as * SPLIT_A_COLS;
            uint32_t part[16];
            if (!wide) {
#pragma unroll
                for (int j = 0; j < 16; ++j) part[j] = __byte_perm(__float_as_uint(v[2 * j]), __float_as_uint(v[2 * j + 1]), 0x7632);
                tc_st16(dst, part);
#pragma unroll
                for (int j = 0; j < 16; ++j) part[j] = 0u;     // another quarter's weights may be wide
                tc_st16(dst + SPLIT_BK / 2, part);
                tc_st16(dst + SPLIT_BK, part);
            } else {
                // hi, mid, lo: each the rounding of what is left
#pragma unroll
                for (int plane = 0; plane < 3; ++plane) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[j] = take_bf16(v[2 * j], v[2 * j + 1]);
                    tc_st16(dst + plane * (SPLIT_BK / 2), part);
                }
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) bad4[j & 3] = fmaf(0.f, v[j], bad4[j & 3]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                s_wide[as][quarter] = wide;
                mbar_arrive(afull + 8 * as);
            }
        }
        const float bad = (bad4[0] + bad4[1]) + (bad4[2] + bad4[3]);
        const bool tiny = (bits & SPLIT_LARGE_BITS) == 0u && ((bits & 0xffffu) != 0u || ((bits & 0x7f800000u) == 0u && (bits & 0x7fffffu) != 0u));
        if (bad != bad || tiny) {
            s_bad[row] = 1.f;
            s_any = 1.f;
        }
    } else if (warp < 12) {
        // ---- sums: a thread has one weight row and half of the tile's rows of x
        const int quarter = warp & 3, half = (warp - 4) >> 2, hn = bn >> 1, wrow = quarter * 32 + lane;
        const int parts = (kb1 - kb0 + SPLIT_GROUP - 1) / SPLIT_GROUP;
        float acc[SPLIT_BN / 2];
#pragma unroll
        for (int j = 0; j < SPLIT_BN / 2; ++j) acc[j] = 0.f;
        fr_pdl_wait();
        for (int j = threadIdx.x - 128; j < bn; j += 256)
            if (m0 + j < p.m && p.marked[m0 + j]) s_any = 1.f;
        bool ok = true;
        const uint32_t src = tmem + ((uint32_t)(quarter * 32) << 16) + half * hn;
        auto add = [&](uint32_t from) {
#pragma unroll
            for (int c = 0; c < SPLIT_BN / 16; c += 2) {       // two loads on their way at a time
                if (8 * c < hn) {
                    float r[8], t[8];
                    const bool both = c + 1 < SPLIT_BN / 16 && 8 * (c + 1) < hn;
                    tc_ld8(from + 8 * c, r);
                    if (both) tc_ld8(from + 8 * c + 8, t);
                    tc_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[8 * c + j] += r[j];
                    if (both) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (8 * c + 8 + j < SPLIT_BN / 2) acc[8 * c + 8 + j] += t[j];
                    }
                }
            }
        };
        for (int part = 0; part < parts; ++part) {
            if (!(ok = mbar_wait(accf, part & 1, p.status, 19))) break;
            tc_fence_after();
            add(src);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acce);
        }
        if (ok && parts > 0) add(src + SPLIT_BN);
        if (ok) {
            // the tile as [row of x][weight row] over the ring of x, which nothing fills any more
            float* part_tile = (float*)x_ring;
#pragma unroll
            for (int j = 0; j < SPLIT_BN / 2; ++j)
                if (j < hn) part_tile[(half * hn + j) * TILE_P + wrow] = acc[j];
        }
    } else {
        if (warp == 12 && elect_one()) {
            // ---- copies
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
            auto load_w = [&](int kb, int s) {
                mbar_expect_tx(wfull + 8 * s, SPLIT_W_BYTES);
                tma_load_2d(smem_u32(smem + s * SPLIT_W_BYTES), &map_w, kb * SPLIT_BK, n0, wfull + 8 * s);
            };
            if (!p.fixed_weights) fr_pdl_wait();
            int early = 0;
            for (; early < SPLIT_W_STAGES && kb0 + early < kb1; ++early) load_w(kb0 + early, early);
            fr_pdl_wait();
            int w_sent = early, x_sent = 0, xs = 0;
            uint32_t x_phase = 1;
            for (int kb = kb0; kb < kb1; ++kb) {
                const int i = kb - kb0, ws = i % SPLIT_W_STAGES;
                if (i >= early) {
                    if (!mbar_wait(wempty + 8 * ws, ((i / SPLIT_W_STAGES) & 1) ^ 1, p.status, 13)) break;
                    load_w(kb, ws);
                    ++w_sent;
                }
                if (!mbar_wait(xempty + 8 * xs, x_phase, p.status, 14)) break;
                mbar_expect_tx(xfull + 8 * xs, x_bytes);
                split_load_3d(smem_u32(x_ring) + xs * x_bytes, &map_x, kb * SPLIT_BK, m0, 0, xfull + 8 * xs);
                ++x_sent;
                if (++xs == XS) { xs = 0; x_phase ^= 1; }
            }
            if (x_sent < kb1 - kb0) {                          // given up: the copies on their way land before the CTA leaves
                for (int i = max(0, w_sent - SPLIT_W_STAGES); i < w_sent; ++i)
                    mbar_wait(wfull + 8 * (i % SPLIT_W_STAGES), (i / SPLIT_W_STAGES) & 1, p.status, 15);
                for (int i = max(0, x_sent - XS); i < x_sent; ++i) mbar_wait(xfull + 8 * (i % XS), (i / XS) & 1, p.status, 15);
            }
        } else if (warp == 13 && elect_one()) {
            // ---- products
            const uint32_t idesc = instr_desc(TILE_P, bn);
            const uint32_t plane = (uint32_t)(bn * SPLIT_BK * 2) >> 4;       // between the planes of x, in descriptor units
            int xs = 0, as = 0;
            uint32_t x_phase = 0, a_phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                const int i = kb - kb0, part = i / SPLIT_GROUP;
                const bool first = i - part * SPLIT_GROUP == 0;
                if (first) {
                    if (!mbar_wait(acce, (part & 1) ^ 1, p.status, 16)) break;
                }
                if (!mbar_wait(xfull + 8 * xs, x_phase, p.status, 17)) break;
                if (!mbar_wait(afull + 8 * as, a_phase, p.status, 18)) break;
                tc_fence_after();
                const volatile int* wv = s_wide[as];
                const bool wide = (wv[0] | wv[1] | wv[2] | wv[3]) != 0;
                const uint32_t large = tmem, small = tmem + SPLIT_BN, wa = tmem + SPLIT_A0 + as * SPLIT_A_COLS;
                const uint64_t xb = smem_desc_64(smem_u32(x_ring) + xs * x_bytes);
#pragma unroll
                for (int s = 0; s < SPLIT_BK / UMMA_K; ++s) {
                    const uint32_t w_hi = wa + 8 * s, w_mid = w_hi + SPLIT_BK / 2, w_lo = w_hi + SPLIT_BK;
                    const uint64_t x_hi = xb + 2 * s, x_mid = x_hi + plane, x_lo = x_mid + plane;
                    tc_mma_tmem_a(large, w_hi, x_hi, idesc, first && s == 0 ? 0u : 1u);
                    tc_mma_tmem_a(small, w_hi, x_lo, idesc, i == 0 && s == 0 ? 0u : 1u);
                    if (wide) {
                        tc_mma_tmem_a(small, w_lo, x_hi, idesc, 1u);
                        tc_mma_tmem_a(small, w_mid, x_mid, idesc, 1u);
                        tc_mma_tmem_a(small, w_mid, x_hi, idesc, 1u);
                    }
                    tc_mma_tmem_a(small, w_hi, x_mid, idesc, 1u);
                }
                tc_commit(xempty + 8 * xs);
                tc_commit(aempty + 8 * as);
                if (i - part * SPLIT_GROUP + 1 == SPLIT_GROUP || kb + 1 == kb1) tc_commit(accf);
                if (++xs == XS) { xs = 0; x_phase ^= 1; }
                if (++as == SPLIT_A_STAGES) { as = 0; a_phase ^= 1; }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 13) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)SPLIT_TMEM) : "memory");
    }
    fr_pdl_wait();
    if (p.splits > 1) fr_cluster_sync();
    const float* tile_sum = (const float*)x_ring;
    float any = s_any;
    for (int s = 0; s < p.splits && p.splits > 1; ++s) any += fr_cluster_load(&s_any, s);
    const bool vec = (p.ldo & 3) == 0 && (((uintptr_t)p.out | (uintptr_t)p.residual) & 15) == 0;
    for (int idx = (split * SPLIT_THREADS + (int)threadIdx.x) * 4; idx < bn * TILE_P; idx += p.splits * SPLIT_THREADS * 4) {
        const int r = idx / TILE_P, c = idx % TILE_P, gm = m0 + r, gn = n0 + c;
        float v[4];
        if (p.splits == 1) {
            const float4 o = *(const float4*)(tile_sum + idx);
            v[0] = o.x; v[1] = o.y; v[2] = o.z; v[3] = o.w;
        } else {
            const float4 f = fr_cluster_load4(tile_sum + idx, 0);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
            for (int s = 1; s < p.splits; ++s) {
                const float4 o = fr_cluster_load4(tile_sum + idx, s);
                v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
            }
        }
        if (gm >= p.m || gn >= p.n) continue;
        const int cols = min(4, p.n - gn);
        if (any != 0.f) {
            const int mark = p.marked[gm];
            for (int j = 0; j < cols; ++j) {
                float b = s_bad[c + j];
                for (int s = 0; s < p.splits && p.splits > 1; ++s) b += fr_cluster_load(s_bad + c + j, s);
                if (mark == SPLIT_BAD || b != 0.f) v[j] = split_plain_dot(p, gm, gn + j);
                else if (mark == SPLIT_TINY) v[j] *= 0x1p-64f;
            }
        }
        const size_t at = (size_t)gm * p.ldo + gn;
        if (vec && cols == 4) {
            if (p.bias.p != nullptr)
                for (int j = 0; j < 4; ++j) v[j] += p.bias.at(gn + j);
            if (p.residual != nullptr) {
                const float4 o = *(const float4*)(p.residual + at);
                v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
            }
            *(float4*)(p.out + at) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            for (int j = 0; j < cols; ++j) {
                float y = v[j];
                if (p.bias.p != nullptr) y += p.bias.at(gn + j);
                if (p.residual != nullptr) y += p.residual[at + j];
                p.out[at + j] = y;
            }
        }
    }
    if (p.splits > 1) fr_cluster_sync();                       // nobody leaves while its shared memory is being read
}

// ------------------------------------------------------------------ host side
typedef CUresult (*SplitEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int split_map(CUtensorMap* map, CUtensorMapDataType type, int dims, const void* base, const cuuint64_t* size, const cuuint64_t* stride,
              const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
    static std::atomic<SplitEncode> known{nullptr};
    SplitEncode enc = known.load(std::memory_order_acquire);
    if (enc == nullptr) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess || ptr == nullptr)
            FR_REFUSE("gemm_simt: the driver does not offer cuTensorMapEncodeTiled");
        enc = (SplitEncode)ptr;
        known.store(enc, std::memory_order_release);
    }
    const cuuint32_t one[3] = {1, 1, 1};
    const CUresult r = enc(map, type, (cuuint32_t)dims, const_cast<void*>(base), size, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) FR_REFUSE("gemm_simt: cuTensorMapEncodeTiled failed with %d", (int)r);
    return FR_OK;
}

long long split_row_bytes(int k) { return 6ll * ((k + 7) / 8 * 8) + 4; }          // a row's planes and its mark
// Rows that `bytes` of scratch hold at a time (0: too few to be worth it).
int split_rows_at_once(int m, int k, long long bytes) {
    const long long rows = (bytes - 16) / split_row_bytes(k);
    if (rows >= m) return m;
    return rows < SPLIT_BN ? 0 : (int)(rows / SPLIT_BN * SPLIT_BN);
}

// CTAs that share a tile's k: the number with the shortest busiest SM.  A CTA's start and end cost as much as some 12 blocks
// of k, a cluster's exchange as 8 more; clusters of a size that no multiple of fills the GPCs leave SMs empty.
int split_k_parts(int tiles, int kb, int sms) {
    const int at_once[9] = {0, sms, sms, sms * 135 / 148, sms * 132 / 148, sms * 130 / 148, sms * 120 / 148, sms * 112 / 148, sms * 112 / 148};
    int best = 1;
    long long best_cost = -1;
    for (int s = 1; s <= 8; ++s) {
        if (s > 1 && kb < 8 * s) break;
        const long long waves = ((long long)tiles * s + at_once[s] - 1) / at_once[s];
        const long long cost = waves * ((kb + s - 1) / s + 12 + (s > 1 ? 8 : 0));
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}

int run_split(SplitArgs p, void* scratch, cudaStream_t stream) {
    const int sms = fr_sm_count() > 0 ? fr_sm_count() : 148;
    const int kp = (p.k + 7) / 8 * 8;
    __nv_bfloat16* planes = (__nv_bfloat16*)scratch;
    int* marked = (int*)((char*)scratch + (6ll * p.m * kp + 15) / 16 * 16);
    p.marked = marked;
    p.tiles_q = (p.m + SPLIT_BN - 1) / SPLIT_BN;
    p.bn = ((p.m + p.tiles_q - 1) / p.tiles_q + 15) / 16 * 16;
    p.x_stages = (SPLIT_MAX_SMEM - SPLIT_FIXED_SMEM) / (3 * p.bn * SPLIT_BK * 2);
    if (p.x_stages > SPLIT_X_STAGES) p.x_stages = SPLIT_X_STAGES;
    const int kb = (p.k + SPLIT_BK - 1) / SPLIT_BK, tiles = (p.n + TILE_P - 1) / TILE_P * p.tiles_q;
    p.splits = split_k_parts(tiles, kb, sms);
    p.kb_per = (kb + p.splits - 1) / p.splits;
    const int smem = SPLIT_FIXED_SMEM + p.x_stages * 3 * p.bn * SPLIT_BK * 2;

    CUtensorMap map_w, map_x;
    const cuuint64_t w_size[2] = {(cuuint64_t)p.k, (cuuint64_t)p.n}, w_stride[1] = {(cuuint64_t)p.ldw * 4};
    const cuuint32_t w_box[2] = {SPLIT_BK, TILE_P};
    int rc = split_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.w, w_size, w_stride, w_box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    const cuuint64_t x_size[3] = {(cuuint64_t)kp, (cuuint64_t)p.m, 3}, x_stride[2] = {(cuuint64_t)kp * 2, (cuuint64_t)kp * 2 * p.m};
    const cuuint32_t x_box[3] = {SPLIT_BK, (cuuint32_t)p.bn, 3};
    rc = split_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, x_size, x_stride, x_box, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;

    static std::atomic<unsigned long long> configured{0};     // devices (as bits) on which the limit has been raised
    int device = 0;
    FR_CUDA(cudaGetDevice(&device));
    if (device < 0 || device >= 64) FR_REFUSE("gemm_simt: device %d is outside the table of 64", device);
    if (!(configured.load(std::memory_order_acquire) & (1ull << device))) {
        FR_CUDA(cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SPLIT_MAX_SMEM));
        configured.fetch_or(1ull << device, std::memory_order_release);
    }
    FR_CUDA(fr_launch(split_rows_kernel, dim3(p.m), dim3(256), 0, stream, p.x, planes, marked, p.m, p.k, kp, p.lda));
    FR_CHECK_LAUNCH("gemm_simt (split rows)");
    FR_CUDA(fr_launch_cluster(gemm_f32_tc_kernel, dim3(tiles * p.splits), dim3(SPLIT_THREADS), smem, stream, (unsigned)p.splits, map_w, map_x, p));
    FR_CHECK_LAUNCH("gemm_simt (tensor cores)");
    return FR_OK;
}

}  // namespace
