// Batched products of at most 16 rows in bfloat16 (the heads' maps of a decode step's rows), mma.sync with float32 sums:
// C[b, m, n] = sum_k A[b, m, k] W[b, n, k].
//
// The weights are read once and the rest is latency, so everything a warp needs is asked for at once: a warp takes 16 weight rows
// (the m side of the MMA; the rows of A are its n side) and up to 128 of K at a time, in 16-byte words straight into registers. An
// MMA's 16 places along K may be any 16 of K as long as both operands agree: lane t of a quad holds entries 8 t .. 8 t + 7 of a run of 32,
// whose first four are its places of one MMA and the others of a second. Weights that the caller holds are asked for before the kernel
// waits for the one before it, which may be what writes others. A chain of MMAs on one accumulator loses a bit or two (the tensor core
// cuts off what a float32 sum would round): each MMA starts from zero and the eight of 128 entries are added as a tree. Results that are
// not the nearest bfloat16, 8 rows of 512 by 128: 4.5e-5 (entries of mean 1: 3.1e-6); a chain 6.3e-5 (2.1e-5), sums by shuffles 4.2e-5
// (3.8e-6). Up to 128 of K a warp walks alone; of a longer K each of the block's four warps takes a quarter, and their sums are added in
// the order of the quarters (16 rows of 64 by 256 3.6 us by warps alone, 1.7 so). The split follows from K alone and a row's sums from its own entries, so its bits do not depend on the
// other rows. Microseconds back to back, 16 maps of 8 rows: 128 x 512 9.5 with a warp per output column and sums by shuffles
// (gemm_simt.cu, which keeps float32 and operands without 16-byte rows) and 1.7, 512 x 128 5.9 and 1.9; 16 rows 13.8 and 2.4, 7.4 and 2.0. A
// decoding layer with these (8 requests of 2,048 keys): 53 and, with the merge of latent_decode.cu, 35.
#include "common.cuh"

namespace {

constexpr int GF_WARPS = 4, GF_RUN = 32, GF_RUNS = 4;      // of K: entries of a run, runs that are asked for at a time

struct FewArgs {
    const bf16* A; const bf16* W; bf16* C;
    int M, N, K;
    long lda, ldw, ldc, batch_a, batch_w, batch_c;
    int held;                                  // 1: no kernel in flight writes W
};

__device__ __forceinline__ void gf_mma(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// MT: tiles of 8 rows of A. QUARTERS: the warps share K (a block has 16 weight rows, else 64).
template <int MT, bool QUARTERS>
__global__ void __launch_bounds__(32 * GF_WARPS) gemm_few_batched_kernel(const FewArgs a) {
    __shared__ float4 shares[QUARTERS ? GF_WARPS : 1][MT][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int n0 = QUARTERS ? blockIdx.x * 16 : (blockIdx.x * GF_WARPS + warp) * 16;
    const int runs = (a.K + GF_RUN - 1) / GF_RUN;
    const int first = QUARTERS ? runs * warp / GF_WARPS : 0, last = QUARTERS ? runs * (warp + 1) / GF_WARPS : runs;
    const bf16* W = a.W + (size_t)blockIdx.y * a.batch_w;
    const bf16* A = a.A + (size_t)blockIdx.y * a.batch_a;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    uint4 w[GF_RUNS][2], x[GF_RUNS][MT];
    auto load_w = [&](int run0) {
#pragma unroll
        for (int i = 0; i < GF_RUNS; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int k = (run0 + i) * GF_RUN + t * 8, n = n0 + g + 8 * r;
                w[i][r] = run0 + i < last && k < a.K && n < a.N ? __ldg(reinterpret_cast<const uint4*>(W + (size_t)n * a.ldw + k)) : none;
            }
    };
    float acc[MT][4] = {};
    if (a.held) load_w(first);
    pdl_wait();
    pdl_trigger();
    if (!a.held) load_w(first);
    for (int run0 = first; run0 < last; run0 += GF_RUNS) {
#pragma unroll
        for (int i = 0; i < GF_RUNS; ++i)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int k = (run0 + i) * GF_RUN + t * 8, row = m * 8 + g;
                x[i][m] = run0 + i < last && k < a.K && row < a.M ? *reinterpret_cast<const uint4*>(A + (size_t)row * a.lda + k) : none;
            }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float part[2 * GF_RUNS][4] = {};
#pragma unroll
            for (int i = 0; i < GF_RUNS; ++i) {
                gf_mma(part[2 * i], w[i][0].x, w[i][1].x, w[i][0].y, w[i][1].y, x[i][m].x, x[i][m].y);
                gf_mma(part[2 * i + 1], w[i][0].z, w[i][1].z, w[i][0].w, w[i][1].w, x[i][m].z, x[i][m].w);
            }
#pragma unroll
            for (int step = 1; step < 2 * GF_RUNS; step *= 2)
#pragma unroll
                for (int i = 0; i < 2 * GF_RUNS; i += 2 * step)
#pragma unroll
                    for (int c = 0; c < 4; ++c) part[i][c] += part[i + step][c];
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[m][c] += part[0][c];
        }
        if (run0 + GF_RUNS < last) load_w(run0 + GF_RUNS);
    }
    if (QUARTERS) {
#pragma unroll
        for (int m = 0; m < MT; ++m) shares[warp][m][lane] = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
        __syncthreads();
        if (warp >= MT) return;                            // warp m finishes the m-th tile of rows
        float4 s = shares[0][warp][lane];
#pragma unroll
        for (int q = 1; q < GF_WARPS; ++q) {
            const float4 v = shares[q][warp][lane];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        acc[0][0] = s.x; acc[0][1] = s.y; acc[0][2] = s.z; acc[0][3] = s.w;
    }
    bf16* C = a.C + (size_t)blockIdx.y * a.batch_c;
#pragma unroll
    for (int m = 0; m < (QUARTERS ? 1 : MT); ++m) {
        const int row = (QUARTERS ? warp : m) * 8 + 2 * t;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int n = n0 + g + 8 * (c >> 1), r = row + (c & 1);
            if (n < a.N && r < a.M) C[(size_t)r * a.ldc + n] = __float2bfloat16_rn(acc[m][c]);
        }
    }
}

}  // namespace

LLMP_API int llmp_gemm_few_batched_supports(const void* A, const void* W, int M, int K, long lda, long ldw, long batch_a, long batch_w) {
    return M > 0 && M <= 16 && K > 0 && (K | lda | ldw | batch_a | batch_w) % 8 == 0 && ((size_t)A | (size_t)W) % 16 == 0;
}

LLMP_API int llmp_gemm_few_batched(const void* A, const void* W, void* C, int batch, int M, int N, int K, long lda, long ldw, long ldc,
                                   long batch_a, long batch_w, long batch_c, int held, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    LLMP_REQUIRE(llmp_gemm_few_batched_supports(A, W, M, K, lda, ldw, batch_a, batch_w) && batch <= 65535,
                 "gemm_few_batched: %d products of %d rows, K %d, or operands without 16-byte rows", batch, M, K);
    const FewArgs a = {(const bf16*)A, (const bf16*)W, (bf16*)C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, held};
    const bool quarters = K > 128;
    const int rows = quarters ? 16 : 16 * GF_WARPS;
    const dim3 grid((unsigned)((N + rows - 1) / rows), batch);
    auto launch = [&](auto kernel) { llmp_launch_dependent(kernel, grid, dim3(32 * GF_WARPS), 0, stream, a); };
    if (M <= 8) quarters ? launch(gemm_few_batched_kernel<1, true>) : launch(gemm_few_batched_kernel<1, false>);
    else quarters ? launch(gemm_few_batched_kernel<2, true>) : launch(gemm_few_batched_kernel<2, false>);
    return llmp_check_launch("gemm_few_batched");
}
