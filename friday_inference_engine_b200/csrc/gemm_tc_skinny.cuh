// The matrix product of a handful of rows with a small matrix: no ring, no tensor memory, no partial tiles in global memory.
//
// What such a product costs on the tcgen05 kernel is a chain of waits: a ring that fills, instructions, partial tiles, their
// counter, their sum.  Here a block owns 16 columns of the output and its warps share k: every lane fetches its pieces of the
// weights with 16-byte loads that are all on their way before the predecessor has finished (fixed weights), then the rows' pieces, multiplies
// with mma.sync.m16n8k16 (the columns on its M side, up to 8 rows on its N side, fp32 sums), and the warps' sums meet in
// shared memory.  A lane's 16 bytes are eight consecutive k; which k an instruction takes from which place is free as long as
// both operands agree, so two instructions take them as they lie.
//
// Included by gemm_tc.cu.
#pragma once

namespace {

constexpr int SKINNY_N = 16;                 // columns per block
constexpr int SKINNY_STEPS = 8;              // pieces of 32 k per warp that are in flight together
constexpr int SKINNY_K = SKINNY_STEPS * 32;  // k per warp and turn

struct SkinnyParams {
    GemmFusion f;                            // the activation's constants, whether the weights are fixed
    const __nv_bfloat16* x;
    const __nv_bfloat16* w;
    void* out;
    const void* bias;
    const void* residual;
    int m, n, k, lda, ldw, ldo, out_dtype, bias_dtype, act;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load_weights(const __nv_bfloat16* p) {       // read once, by one block
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// MT: groups of 8 rows
template <int WARPS, int MT>
__global__ void __launch_bounds__(32 * WARPS, WARPS == 8 ? 2 : 1)
gemm_skinny_kernel(const SkinnyParams p) {
    __shared__ float red[WARPS][MT * 8][SKINNY_N + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * SKINNY_N;
    const __nv_bfloat16* wl = p.w + (size_t)min(n0 + g, p.n - 1) * p.ldw;
    const __nv_bfloat16* wh = p.w + (size_t)min(n0 + g + 8, p.n - 1) * p.ldw;
    const __nv_bfloat16* xr[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) xr[i] = p.x + (size_t)min(i * 8 + g, p.m - 1) * p.lda;
    fr_pdl_launch();
    if (!p.f.fixed_weights) fr_pdl_wait();
    float acc[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const uint4 none = make_uint4(0, 0, 0, 0);
    for (int k0 = warp * SKINNY_K; k0 < p.k || k0 < WARPS * SKINNY_K; k0 += WARPS * SKINNY_K) {
        uint4 lo[SKINNY_STEPS], hi[SKINNY_STEPS];
#pragma unroll
        for (int s = 0; s < SKINNY_STEPS; ++s) {
            const int k = k0 + s * 32 + t * 8;
            lo[s] = hi[s] = none;
            if (k < p.k) {
                lo[s] = load_weights(wl + k);
                hi[s] = load_weights(wh + k);
            }
        }
        if (k0 < WARPS * SKINNY_K) fr_pdl_wait();        // fixed weights do not depend on the kernel before this one; the rows do
#pragma unroll
        for (int s = 0; s < SKINNY_STEPS; ++s) {
            const int k = k0 + s * 32 + t * 8;
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const uint4 b = k < p.k ? *(const uint4*)(xr[i] + k) : none;
                mma_16816(acc[i], lo[s].x, hi[s].x, lo[s].y, hi[s].y, b.x, b.y);
                mma_16816(acc[i], lo[s].z, hi[s].z, lo[s].w, hi[s].w, b.z, b.w);
            }
        }
    }
    // lane (g, t) has columns g and g + 8 of rows 2 t and 2 t + 1
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) red[warp][i * 8 + 2 * t + (j & 1)][g + (j & 2) * 4] = acc[i][j];
    __syncthreads();
    const bool gated = p.act >= 1 && p.act <= 3;
    for (int idx = threadIdx.x; idx < (gated ? MT * 64 : MT * 128); idx += 32 * WARPS) {
        const int row = gated ? idx / 8 : idx / 16, c = gated ? idx % 8 * 2 : idx % 16;
        if (row >= p.m || n0 + c >= p.n) continue;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) v += red[w][row][c];
        if (gated) {
            float u = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) u += red[w][row][c + 1];
            ((__nv_bfloat16*)p.out)[(size_t)row * p.ldo + ((n0 + c) >> 1)] = __float2bfloat16_rn(gated_mul(p, v, u));
            continue;
        }
        if (p.act == ACT_RELU_SQUARED) {
            v = fmaxf(v, 0.f);
            v *= v;
        }
        const size_t at = (size_t)row * p.ldo + n0 + c;
        if (p.bias != nullptr) v += bias_at(p, n0 + c);
        if (p.out_dtype == FR_BF16) {
            if (p.residual != nullptr) v += __bfloat162float(((const __nv_bfloat16*)p.residual)[at]);
            ((__nv_bfloat16*)p.out)[at] = __float2bfloat16_rn(v);
        } else {
            if (p.residual != nullptr) v += ((const float*)p.residual)[at];
            ((float*)p.out)[at] = v;
        }
    }
}

template <int WARPS, int MT>
int launch_skinny(const SkinnyParams& p, cudaStream_t stream) {
    FR_CUDA(fr_launch(gemm_skinny_kernel<WARPS, MT>, dim3((p.n + SKINNY_N - 1) / SKINNY_N), dim3(32 * WARPS), 0, stream, p));
    FR_CHECK_LAUNCH("gemm_tc (skinny)");
    return FR_OK;
}

}  // namespace
