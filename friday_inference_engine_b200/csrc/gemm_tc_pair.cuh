// The matrix product of many rows on pairs of SMs: two CTAs of a cluster share one 256 x bn tile
// (tcgen05.mma.cta_group::2).  Each CTA loads its own 128 rows of the activations and HALF of the tile's weight
// rows; the instruction, issued by the pair's first CTA, reads both halves.  Per 128 x bn of output a CTA then
// moves 16 KB + bn * 64 bytes per k block into shared memory instead of 16 KB + bn * 128: the product of a
// prompt is bound by exactly that traffic and by the power it costs.
//
// Included by gemm_tc.cu (after its parameter structs and epilogue helpers); rows on the M side only, every tile
// computed whole (no split of k).  The protocol between the two CTAs:
//   * stage s of the ring is filled by both CTAs' TMA warps; all four loads signal the FIRST CTA's full[s], which
//     expects the bytes of both;
//   * the first CTA's MMA thread waits for full[s], issues the instructions, and commits to empty[s] of BOTH CTAs
//     (a multicast commit), after a tile's last k block to acc_full[a] of both;
//   * both CTAs' epilogue warps read their own 128 lanes of the accumulator and arrive on the FIRST CTA's
//     acc_empty[a] (sixteen arrivals).
// Every wait is bounded as in gemm_tc.cu.  Neither CTA leaves before the other (a cluster barrier before tensor
// memory is freed): a CTA's shared memory and barriers are written from outside until the pair is done.
#pragma once

namespace {

constexpr int PAIR_BN = 256;                          // widest tile; p.bn may be any multiple of 16 up to it
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_Q_BYTES = (PAIR_BN / 2) * TILE_K * 2;
constexpr int PAIR_STAGE_BYTES = P_BYTES + PAIR_Q_BYTES;
constexpr int PAIR_SMEM_BYTES = PAIR_STAGES * PAIR_STAGE_BYTES + 1024 + (2 * PAIR_STAGES + 4) * 8 + 64 + PAIR_BN * 4 + TILE_P * 4;
// Eight warps finish a tile, two to each quarter of the accumulator's lanes, which take its groups of 16 columns in turn (with a norm
// begun: a half each): with one per quarter a gated tile's epilogue was longer than its products where k is short (2048 x 12288 x
// 2048: 107 us with one, 70 with two; eight experts of some 512 rows, x 4096 x 2048: 113 and 70 to 76; a prompt of 2,048 rows of the
// 7B shape 5 % less).
constexpr int PAIR_FINISHERS = 256, PAIR_THREADS = 64 + PAIR_FINISHERS;

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}
// `bar` is a shared::cluster address: the barrier may be the other CTA's.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives, once the instructions issued so far are done, on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}

// Row tiles of a group.  Every group reads all weights again, so wide outputs want groups as high as L2 keeps their rows
// (17971 x 37888 x 3584, TFLOP/s at 4 / 8 / 12 / 16 / 24 row tiles: 1,304 / 1,353 / 1,373 / 1,372 / 1,364; 4096 rows: 1,310 /
// 1,344 / 1,345 / 1,379 with all 16 in one).  Where the columns are so few that a handful of row tiles keeps every pair busy,
// higher groups only spread the rows that are in use (17971 x 3584 x 18944: 1,308 / 1,305 / 1,284 / 1,287 / 1,222, x 4608 x
// 3584: 1,347 / 1,326 / 1,315 / 1,316 / 1,304).  The groups are made alike.
inline int pair_group(int tiles_p, int tiles_q, int pairs) {
    int high = 16;
    if (2 * tiles_q < pairs) high = (pairs + tiles_q - 1) / tiles_q < 4 ? 4 : (pairs + tiles_q - 1) / tiles_q;
    const int groups = (tiles_p + high - 1) / high;
    return (tiles_p + groups - 1) / groups;
}

// Where a tile lies.  Row tiles go in groups of p.group_p: a group's row tiles run fastest, then its columns, then the next
// group, so that the 74 tiles that are computed at a time find each other's operands in L2.  With all row tiles in one group
// a prompt batch of 17,971 rows read its activations (130 MB at k = 3584, as much as L2 holds) again for every column tile:
// 17971 x 37888 x 3584 ran at 1,106 TFLOP/s under the power cap, 1,372 with groups of 16 (cuBLAS: 1,386).
__device__ __forceinline__ void pair_tile(const GemmParams& p, int tile, int& p_blk, int& q_blk) {
    const int group = tile / (p.group_p * p.tiles_q), first = group * p.group_p;
    const int high = min(p.group_p, p.tiles_p - first), at = tile - first * p.tiles_q;
    q_blk = at / high;
    p_blk = first + at - q_blk * high;
}

__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

// The tiles of one pair, in the order in which all three roles walk them.  GROUPED: the rows are groups (rows off[g] to
// off[g + 1] - 1), each with weights of its own; a group's row tiles start at its first row, and its tiles lie together.
template <bool GROUPED>
struct PairWalk {
    const GemmParams& p;
    const int* off;
    int tile, step, group, base;               // base: the group's first tile
    int row0, row_end, q_blk;                  // the tile's first row, where its rows end, its column tile
    __device__ PairWalk(const GemmParams& p_, const int* off_, int pair, int pairs)
        : p(p_), off(off_), tile(pair - pairs), step(pairs), group(0), base(0), row0(0), row_end(p_.p_rows), q_blk(0) {}
    __device__ bool next() {
        tile += step;
        if constexpr (GROUPED) {
            int high = 0;
            for (;; ++group) {
                if (group >= p.groups) return false;
                high = (off[group + 1] - off[group] + 2 * TILE_P - 1) / (2 * TILE_P);
                if (tile < base + high * p.tiles_q) break;
                base += high * p.tiles_q;
            }
            const int at = tile - base;
            q_blk = at / high;
            row0 = off[group] + (at - q_blk * high) * (2 * TILE_P);
            row_end = off[group + 1];
        } else {
            if (tile >= p.dp_tiles) return false;
            int p_blk;
            pair_tile(p, tile, p_blk, q_blk);
            row0 = p_blk * (2 * TILE_P);
        }
        return true;
    }
};

constexpr int MAX_GROUPS = 256;

template <bool GROUPED>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q, const GemmParams p) {
    __shared__ int s_off[GROUPED ? MAX_GROUPS + 1 : 1];
    constexpr int STAGES = PAIR_STAGES, STAGE_BYTES = PAIR_STAGE_BYTES, BN = PAIR_BN;
    constexpr int TMEM_COLS = 2 * BN;
    const int bn = p.bn, half = bn >> 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    // bars: full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 4);
    volatile int* s_gave_up = (volatile int*)(tmem_slot + 1);               // a finisher of this CTA has stopped waiting
    float* s_gw = (float*)((uint8_t*)(bars + 2 * STAGES + 4) + 64);         // [BN] norm weights of the tile's columns
    float* s_ss = s_gw + BN;                                                // [128] the rows' sums of squares over a tile's first half
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = fr_cluster_rank();                                 // 0: the CTA that issues the instructions
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const uint32_t accf0 = smem_u32(bars + 2 * STAGES), acce0 = smem_u32(bars + 2 * STAGES + 2);
    const uint32_t first_full0 = cluster_addr(full0, 0), first_acce0 = cluster_addr(acce0, 0);

    if (threadIdx.x == 0) {
        *s_gave_up = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(accf0 + 8 * a, 1);
            mbar_init(acce0 + 8 * a, 2 * PAIR_FINISHERS / 32);      // the epilogue warps of both CTAs
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"((uint32_t)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if constexpr (GROUPED) {                               // where the groups lie is the predecessor's result
        fr_pdl_wait();
        for (int g = threadIdx.x; g <= p.groups; g += PAIR_THREADS) s_off[g] = p.group_rows != nullptr ? p.group_rows[g] : g * p.group_size;
    }
    tc_fence_before();
    __syncthreads();
    fr_cluster_sync();                                     // the other CTA's barriers are ready before anything reaches them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) fr_pdl_launch();

    if (warp == 0) {
        if (elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_p) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
            struct Walk {                                  // the k blocks this pair will load, in order
                PairWalk<GROUPED> tiles;
                int kb;
                bool live;
                __device__ Walk(const GemmParams& pp, const int* off, int cta, int grid) : tiles(pp, off, cta, grid), kb(0) { live = tiles.next(); }
                __device__ void step() {
                    if (++kb >= tiles.p.kb_total) {
                        kb = 0;
                        live = tiles.next();
                    }
                }
            };
            auto load_weights = [&](const Walk& at, uint32_t dst, uint32_t bar) {
                const int row = at.tiles.q_blk * bn + (int)rank * half;
                if constexpr (GROUPED) tma_load_3d_pair(dst, &map_q, at.kb * TILE_K, row, at.tiles.group, bar);
                else tma_load_2d_pair(dst, &map_q, at.kb * TILE_K, row, bar);
            };
            // Fixed weights do not depend on the kernel before this one; the activations do.  Fill the ring with
            // weight slices first, then wait for the predecessor, then add the activation slices.
            if (!p.f.fixed_weights) fr_pdl_wait();
            const uint32_t stage_tx = 2u * (P_BYTES + (uint32_t)half * TILE_K * 2);      // both CTAs' bytes of a stage
            Walk head(p, s_off, pair, pairs);
            Walk ahead(p, s_off, pair, pairs);
            int early = 0;
            for (; early < STAGES && ahead.live; ++early, ahead.step()) {
                if (rank == 0) mbar_expect_tx(full0 + 8 * early, stage_tx);
                load_weights(ahead, smem_u32(smem + early * STAGE_BYTES) + P_BYTES, first_full0 + 8 * early);
            }
            fr_pdl_wait();
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (; head.live && ok; head.step()) {
                const uint32_t dst = smem_u32(smem + stage * STAGE_BYTES);
                if (early > 0) {
                    --early;                                 // the weight slice of this stage is already on its way
                } else {
                    if (!(ok = mbar_wait(empty0 + 8 * stage, phase ^ 1, p.status, 1))) break;
                    if (rank == 0) mbar_expect_tx(full0 + 8 * stage, stage_tx);
                    load_weights(head, dst + P_BYTES, first_full0 + 8 * stage);
                }
                const int row = head.tiles.row0 + (int)rank * TILE_P;
                if (GROUPED && p.x_planes)
                    tma_load_3d_pair(dst, &map_p, head.kb * TILE_K, row - s_off[head.tiles.group], head.tiles.group, first_full0 + 8 * stage);
                else tma_load_2d_pair(dst, &map_p, head.kb * TILE_K, row, first_full0 + 8 * stage);
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            fr_pdl_wait();
            const uint32_t idesc = instr_desc(2 * TILE_P, bn);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int it = 0;
            PairWalk<GROUPED> tiles(p, s_off, pair, pairs);
            for (; ok && tiles.next(); ++it) {
                const int a = it & 1;
                const uint32_t acc_phase = (it >> 1) & 1;
                if (!(ok = mbar_wait(acce0 + 8 * a, acc_phase ^ 1, p.status, 2))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + a * BN;
                for (int kb = 0; kb < p.kb_total; ++kb) {
                    if (!(ok = mbar_wait(full0 + 8 * stage, phase, p.status, 3))) break;
                    tc_fence_after();
                    const uint32_t pa = smem_u32(smem + stage * STAGE_BYTES);
                    const uint64_t da = smem_desc(pa), db = smem_desc(pa + P_BYTES);
#pragma unroll
                    for (int k = 0; k < TILE_K / UMMA_K; ++k)
                        tc_mma_pair(d_tmem, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit_pair(empty0 + 8 * stage);   // the stage is free in both CTAs once these products are done
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (ok) tc_commit_pair(accf0 + 8 * a);    // the accumulator is complete, in both CTAs
            }
        }
    } else {
        const int quarter = warp & 3;                      // TMEM lanes this warp may read: 32*quarter ..
        const int i_local = quarter * 32 + lane;
        const int et = threadIdx.x - 64;                   // 0..255 among the epilogue threads
        const int share = et >> 7;                         // which of the quarter's two warps
        fr_pdl_wait();
        bool ok = true;
        int it = 0;
        const GemmFusion& f = p.f;
        const bool norm_rows = f.norm_out != nullptr;
        int scale_row = -1;
        float row_scale = 1.f;
        PairWalk<GROUPED> tiles(p, s_off, pair, pairs);
        for (; ok && tiles.next(); ++it) {
            const int q_blk = tiles.q_blk, gi = tiles.row0 + (int)rank * TILE_P + i_local;
            const int a = it & 1;
            const uint32_t acc_phase = (it >> 1) & 1;
            if (f.in_ssq != nullptr && gi != scale_row) {
                // the deferred norm of the input: the factor of this thread's row
                float ss = 0.f;
                if (gi < p.p_rows)
                    for (int t = 0; t < f.in_parts; ++t) ss += __ldcg(f.in_ssq + (size_t)t * p.p_rows + gi);
                row_scale = 1.0f / sqrtf(ss / f.in_width + f.in_eps);
                scale_row = gi;
            }
            if (norm_rows) {
                asm volatile("bar.sync 1, 256;" ::: "memory");
                for (int i = et; i < bn; i += PAIR_FINISHERS) {
                    const int col = q_blk * bn + i;
                    s_gw[i] = col >= p.q_rows ? 0.f : f.norm_w_dtype == FR_F32 ? ((const float*)f.norm_w)[col]
                                                                               : __bfloat162float(((const __nv_bfloat16*)f.norm_w)[col]);
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            ok = mbar_wait(accf0 + 8 * a, acc_phase, p.status, 4);
            if (norm_rows) {                               // these warps meet again below: they go on, or leave, together
                if (!ok) *s_gave_up = 1;
                asm volatile("bar.sync 1, 256;" ::: "memory");
                ok = *s_gave_up == 0;
            }
            if (!ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + a * BN;
            auto sums16 = [&](int c, float (&v)[16]) {
                uint32_t r[16];
                tc_ld16(taddr + c * 16, r);
                tc_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                if (f.in_ssq != nullptr)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] *= row_scale;
            };
            // With a norm begun, a row's two warps have its columns' first and second half: the second adds its squares to
            // the sum of the first, so that a row's sum has the order that it has everywhere (its values wait in registers).
            uint32_t kept[GROUPED ? 1 : PAIR_BN / 32][8];
            if (!GROUPED && norm_rows) {
                const int first = (bn / 16 + 1) / 2, c0 = share == 0 ? 0 : first, c1 = share == 0 ? first : bn / 16;
#pragma unroll
                for (int i = 0; i < (GROUPED ? 1 : PAIR_BN / 32); ++i) {
                    const int c = c0 + i;
#pragma unroll
                    for (int j = 0; j < 8; ++j) kept[i][j] = 0u;
                    if (c < c1) {
                        float v[16];
                        sums16(c, v);
                        finish16_scaled(p, s_gw + c * 16, gi, q_blk * bn + c * 16, v, kept[i], false);
                    }
                }
            } else {
#pragma unroll 1
                for (int c = share; c < bn / 16; c += 2) {
                    float v[16];
                    sums16(c, v);
                    if (!GROUPED || gi < tiles.row_end) finish16(p, gi, q_blk * bn + c * 16, v);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(first_acce0 + 8 * a);     // the accumulator may be overwritten
            if (!GROUPED && norm_rows) {
                float ss = 0.f;
                if (share == 0) {
#pragma unroll
                    for (int i = 0; i < (GROUPED ? 1 : PAIR_BN / 32); ++i) add_squares(kept[i], ss);
                    s_ss[i_local] = ss;
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (share == 1) {
                    ss = s_ss[i_local];
#pragma unroll
                    for (int i = 0; i < (GROUPED ? 1 : PAIR_BN / 32); ++i) add_squares(kept[i], ss);
                    if (gi < p.p_rows) f.out_ssq[(size_t)q_blk * p.p_rows + gi] = ss;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    fr_cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                     : "memory");
    }
}

}  // namespace
