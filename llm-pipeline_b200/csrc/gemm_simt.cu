// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) on the CUDA cores with float32 accumulation.
// This is the matrix product of the true 32-bit path (no tensor core, no reduced-precision
// mode) and accepts every size. Each output element adds its K products in ascending k (of a narrow matrix with a long K: those of
// each segment of K, and the segments' sums in their order; which it is follows from the matrix alone), so a row's result does not
// depend on how many other rows are in the call.
#include "common.cuh"

int llmp_sm_count();

namespace {

// Four consecutive entries of a row from k on; entries from K on are 0. VEC: 4-entry pieces are aligned and K is a multiple of 4.
template <bool VEC> __device__ __forceinline__ float4 gt_load4(const float* row, int k, int K) {
    if (VEC) return k < K ? *reinterpret_cast<const float4*>(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(k < K ? row[k] : 0.f, k + 1 < K ? row[k + 1] : 0.f, k + 2 < K ? row[k + 2] : 0.f, k + 3 < K ? row[k + 3] : 0.f);
}
template <bool VEC> __device__ __forceinline__ float4 gt_load4(const bf16* row, int k, int K) {
    if (VEC) {
        if (k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
        const uint2 raw = *reinterpret_cast<const uint2*>(row + k);
        const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&raw);
        return make_float4(__low2float(v[0]), __high2float(v[0]), __low2float(v[1]), __high2float(v[1]));
    }
    return make_float4(k < K ? to_float(row[k]) : 0.f, k + 1 < K ? to_float(row[k + 1]) : 0.f, k + 2 < K ? to_float(row[k + 2]) : 0.f,
                       k + 3 < K ? to_float(row[k + 3]) : 0.f);
}

// A block makes BM x BN outputs with TM x TN of them a thread. BK entries of K at a time lie in shared memory as rows padded by 4
// (a quarter-warp's 16-byte reads of consecutive rows meet no bank twice), in two buffers, one barrier for each; those of the next
// AHEAD are on their way in registers. A thread reads 4 entries of K of its TM + TN rows as 16-byte words for 4 TM TN multiply-adds.
// CLUSTER: K is cut into segments, a block of a cluster for each. They leave their sums in shared memory, and each adds up a share of the
// tile from all of them.
template <typename TI, typename TO, int BM, int BN, int BK, int TM, int TN, int AHEAD, bool VEC, bool CLUSTER>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_nt_kernel(const TI* __restrict__ A, const TI* __restrict__ W, const void* __restrict__ bias, int bias_bf16,
               TO* __restrict__ C, int M, int N, int K, long lda, long ldw, long ldc, long batch_a, long batch_w, long batch_c, int segment) {
    constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY, QUADS = BK / 4, LD = BK + 4;
    constexpr int LA = BM * QUADS / THREADS, LW = BN * QUADS / THREADS;      // 4-entry pieces of each operand a thread brings
    static_assert(LA * THREADS == BM * QUADS && LW * THREADS == BN * QUADS, "the pieces of a tile are shared out evenly");
    // blockIdx.z counts the products of a batch: each has its own A, W and C, the given strides apart
    // (of a cluster the blocks are neighbours along x, where a grid may be long: a batch with its segments may be more than 65,535)
    const int segments = CLUSTER ? (K + segment - 1) / segment : 1, rank = CLUSTER ? (int)blockIdx.x % segments : 0;
    A += (size_t)blockIdx.z * batch_a;
    W += (size_t)blockIdx.z * batch_w;
    C += (size_t)blockIdx.z * batch_c;
    if (CLUSTER) {                                 // this block's part of K
        A += (size_t)rank * segment;
        W += (size_t)rank * segment;
        K = min(segment, K - rank * segment);
    }
    __shared__ __align__(16) float operands[2 * (BM + BN) * LD];
    float (*const As)[BM * LD] = reinterpret_cast<float (*)[BM * LD]>(operands);
    float (*const Ws)[BN * LD] = reinterpret_cast<float (*)[BN * LD]>(operands + 2 * BM * LD);
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = (int)blockIdx.x / segments * BN;
    float acc[TM][TN] = {};
    float4 ra[AHEAD][LA], rw[AHEAD][LW];
    auto fetch = [&](int k0, float4 (&pa)[LA], float4 (&pw)[LW]) {           // past the end of K: zeros, without a read
#pragma unroll
        for (int r = 0; r < LA; ++r) {
            const int e = tid + r * THREADS, m = m0 + e / QUADS;
            pa[r] = m < M ? gt_load4<VEC>(A + (size_t)m * lda, k0 + e % QUADS * 4, K) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < LW; ++r) {
            const int e = tid + r * THREADS, n = n0 + e / QUADS;
            pw[r] = n < N ? gt_load4<VEC>(W + (size_t)n * ldw, k0 + e % QUADS * 4, K) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto keep = [&](int buffer, const float4 (&pa)[LA], const float4 (&pw)[LW]) {
#pragma unroll
        for (int r = 0; r < LA; ++r) {
            const int e = tid + r * THREADS;
            *reinterpret_cast<float4*>(&As[buffer][e / QUADS * LD + e % QUADS * 4]) = pa[r];
        }
#pragma unroll
        for (int r = 0; r < LW; ++r) {
            const int e = tid + r * THREADS;
            *reinterpret_cast<float4*>(&Ws[buffer][e / QUADS * LD + e % QUADS * 4]) = pw[r];
        }
    };
    auto multiply = [&](int buffer) {
#pragma unroll
        for (int q = 0; q < QUADS; ++q) {
            float4 a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(&As[buffer][(ty + i * TY) * LD + q * 4]);
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(&Ws[buffer][(tx + j * TX) * LD + q * 4]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    };
#pragma unroll
    for (int d = 0; d < AHEAD; ++d) fetch(d * BK, ra[d], rw[d]);
    const int steps = (K + BK - 1) / BK;
    for (int i0 = 0; i0 < steps; i0 += AHEAD) {
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) {
            const int i = i0 + d;
            if (i >= steps) break;
            keep(i & 1, ra[d], rw[d]);                         // everyone left this buffer a barrier ago
            __syncthreads();
            fetch((i + AHEAD) * BK, ra[d], rw[d]);
            multiply(i & 1);
        }
    }
    if (CLUSTER) {
        constexpr int PITCH = BN + 1;
        static_assert(BM * PITCH <= 2 * (BM + BN) * LD, "a tile's sums take the operands' place");
        float* sums = operands;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) sums[(ty + i * TY) * PITCH + tx + j * TX] = acc[i][j];
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        const unsigned own = (unsigned)__cvta_generic_to_shared(sums);
        for (int e = rank * THREADS + tid; e < BM * BN; e += segments * THREADS) {
            const int m = m0 + e / BN, n = n0 + e % BN;
            if (m >= M || n >= N) continue;
            const unsigned at = own + (unsigned)(e / BN * PITCH + e % BN) * 4u;
            float v = 0.f;
            for (int q = 0; q < segments; ++q) {
                unsigned there;
                float s;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(there) : "r"(at), "r"(q));
                asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(s) : "r"(there) : "memory");
                v = q ? v + s : s;
            }
            if (bias) v += load_as_float(bias, bias_bf16, n);
            C[(size_t)m * ldc + n] = from_float<TO>(v);
        }
        // nobody leaves while another block reads its sums (a warp's lanes, which have shares of different lengths, arrive as one)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * TY;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * TX;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += load_as_float(bias, bias_bf16, n);
            C[(size_t)m * ldc + n] = from_float<TO>(v);
        }
    }
}

// Few weight rows with a long K leave SMs idle up to thousands of rows, so K is cut into up to as many segments as a cluster may have
// blocks. 96 x 2,048, microseconds with a whole K in a block and in segments: 1 row 39 and 8, 203 rows 39 and 14, 2,048 rows 54 and 39, 8,192 156
// and 149, 40,000 646 and 695. Whether K is cut may not depend on the rows, and of wider matrices fewer rows fill the chip, where
// segments are slower: 2,048 and 8,192 rows, K 2,048, 128 columns 54 and 40, 156 and 151; 160 columns 74 and 76, 198 and 223; 256 columns
// 84 and 78, 219 and 297; 1,024 columns 219 and 297, 862 and 1,136.
constexpr int GT_SEGMENT = 256, GT_MAX_SEGMENTS = 8, GT_NARROW = 128;
int gt_segment(int N, int K, bool float32) {
    const int most = (K + GT_SEGMENT - 1) / GT_SEGMENT, count = most < GT_MAX_SEGMENTS ? most : GT_MAX_SEGMENTS;
    return N > GT_NARROW || !float32 ? K : ((K + count - 1) / count + 31) / 32 * 32;
}

// Shared memory delivers a thread's words at 128 bytes a clock and SM whether lanes ask for the same or not, so a tile's speed is
// its multiply-adds per word read: 8 x 8 outputs a thread make 42 TFLOP/s (700 x 6,144 x 2,048; 4 x 4 made 31, and 4-byte reads
// of a single buffer 21), but their blocks of two warps need three an SM. Fewer blocks, smaller tiles, so that every SM has
// one; and where even the smallest leave SMs idle, more threads a tile for the latency. 203 rows, microseconds before and now:
// 4,096 x 1,024 114 -> 77, 1,024 x 2,048 148 -> 53; 1 row, 1,024 x 1,024 74 -> 18; 2,048 rows, 4,096 x 4,096 2,951 -> 1,708.
template <typename TI, typename TO, bool VEC>
void launch_nt(const TI* A, const TI* W, const void* bias, int bias_bf16, TO* C, int batch, int M, int N, int K, long lda, long ldw, long ldc,
               long batch_a, long batch_w, long batch_c, cudaStream_t stream) {
    const long sms = llmp_sm_count();
    const int segment = gt_segment(N, K, sizeof(TI) == 4), segments = (K + segment - 1) / segment;
    auto blocks = [&](int bm, int bn) { return (long)((N + bn - 1) / bn) * ((M + bm - 1) / bm) * batch; };
    auto launch = [&](auto kernel, int bm, int bn, int threads, bool cluster) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3((unsigned)((N + bn - 1) / bn * (cluster ? segments : 1)), (M + bm - 1) / bm, batch);
        config.blockDim = dim3(threads);
        config.stream = stream;
        cudaLaunchAttribute attr[1];                           // (not a dependent launch: blocks that begin before the last kernel's have
        attr[0].id = cudaLaunchAttributeClusterDimension;      // ended crowd on the SMs that are free first, 250 -> 302 us a layer)
        attr[0].val.clusterDim.x = segments;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        config.attrs = attr;
        config.numAttrs = cluster ? 1 : 0;
        cudaLaunchKernelEx(&config, kernel, A, W, bias, bias_bf16, C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, segment);
    };
#define LLMP_NT(BM, BN, BK, TM, TN, AHEAD, SEG) \
    launch(gemm_nt_kernel<TI, TO, BM, BN, BK, TM, TN, AHEAD, VEC, SEG>, BM, BN, (BM / TM) * (BN / TN), SEG)
    if constexpr (sizeof(TI) == 4) {
        if (segments > 1) {
            if (blocks(64, 64) * segments >= 2 * sms) LLMP_NT(64, 64, 32, 8, 8, 1, true);
            else if (blocks(32, 32) * segments >= sms) LLMP_NT(32, 32, 32, 4, 4, 1, true);
            else LLMP_NT(32, 32, 32, 2, 2, 2, true);
            return;
        }
    }
    if (blocks(64, 64) >= 3 * sms) LLMP_NT(64, 64, 32, 8, 8, 1, false);
    else if (blocks(64, 64) >= sms) LLMP_NT(64, 64, 16, 8, 4, 1, false);
    else if (blocks(32, 32) >= sms) LLMP_NT(32, 32, 32, 4, 4, 1, false);
    else LLMP_NT(32, 32, 32, 2, 2, 2, false);
#undef LLMP_NT
}

template <typename TI, typename TO>
void launch_nt_types(const void* A, const void* W, const void* bias, int bias_bf16, void* C, int batch, int M, int N, int K, long lda, long ldw,
                     long ldc, long batch_a, long batch_w, long batch_c, cudaStream_t stream) {
    const size_t piece = 4 * sizeof(TI);
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0 && ((size_t)A | (size_t)W) % piece == 0;
    if (vec) launch_nt<TI, TO, true>((const TI*)A, (const TI*)W, bias, bias_bf16, (TO*)C, batch, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, stream);
    else launch_nt<TI, TO, false>((const TI*)A, (const TI*)W, bias, bias_bf16, (TO*)C, batch, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, stream);
}

// false: no such combination of types
bool launch_nt_any(const void* A, const void* W, const void* bias, int bias_bf16, void* C, int in_dtype, int out_dtype, int batch, int M, int N,
                   int K, long lda, long ldw, long ldc, long batch_a, long batch_w, long batch_c, cudaStream_t stream) {
#define LLMP_NT_TYPES(TI, TO) launch_nt_types<TI, TO>(A, W, bias, bias_bf16, C, batch, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, stream)
    if (in_dtype == LLMP_F32 && out_dtype == LLMP_F32) LLMP_NT_TYPES(float, float);
    else if (in_dtype == LLMP_BF16 && out_dtype == LLMP_BF16) LLMP_NT_TYPES(bf16, bf16);
    else if (in_dtype == LLMP_BF16 && out_dtype == LLMP_F32) LLMP_NT_TYPES(bf16, float);
    else return false;
#undef LLMP_NT_TYPES
    return true;
}

}  // namespace

#define GT_MAX_ROWS (65535 * 64)      // what a grid can hold of the tiles of 64 rows, which so many rows take whatever N is

// in_dtype: type of A and W.  out_dtype: type of C (float32, or the input type).
LLMP_API int llmp_gemm_simt(const void* A, const void* W, const void* bias, int bias_dtype, void* C, int in_dtype,
                            int out_dtype, int M, int N, int K, long lda, long ldw, long ldc, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    LLMP_REQUIRE(K > 0, "gemm: bad K %d", K);
    LLMP_REQUIRE(M <= GT_MAX_ROWS, "gemm: too many rows %d", M);
    if (!launch_nt_any(A, W, bias, bias_dtype == LLMP_BF16, C, in_dtype, out_dtype, 1, M, N, K, lda, ldw, ldc, 0, 0, 0, stream)) {
        llmp_set_error("gemm: unsupported type combination in=%d out=%d", in_dtype, out_dtype);
        return 1;
    }
    return llmp_check_launch("gemm_simt");
}

// A batch of products of at most 16 rows each (a decode step), float32 or without 16-byte rows (else gemm_few_batched.cu): a warp per output column reads the column's weight
// row once and keeps one sum per row of A; the K products of a sum are added lane by lane in ascending k, then across
// the lanes in a fixed order.
#define GR_MAX_ROWS 16
__device__ __forceinline__ void gr_load8(const bf16* p, float (&v)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __low2float(h2[i]);
        v[2 * i + 1] = __high2float(h2[i]);
    }
}
__device__ __forceinline__ void gr_load8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// VEC: K, the strides and the addresses allow 16-byte loads of 8 consecutive entries.
template <typename TI, typename TO, bool VEC>
__global__ void __launch_bounds__(256)
gemm_rows_kernel(const TI* __restrict__ A, const TI* __restrict__ W, TO* __restrict__ C, int M, int N, int K, long lda, long ldw,
                 long ldc, long batch_a, long batch_w, long batch_c) {
    const int lane = threadIdx.x & 31;
    const int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (n >= N) return;
    A += (size_t)blockIdx.y * batch_a;
    C += (size_t)blockIdx.y * batch_c;
    const TI* w = W + (size_t)blockIdx.y * batch_w + (size_t)n * ldw;
    float acc[GR_MAX_ROWS];
#pragma unroll
    for (int m = 0; m < GR_MAX_ROWS; ++m) acc[m] = 0.f;
    if (VEC) {
        for (int k = lane * 8; k < K; k += 256) {
            float wv[8];
            gr_load8(w + k, wv);
#pragma unroll
            for (int m = 0; m < GR_MAX_ROWS; ++m) {
                if (m < M) {
                    float xv[8];
                    gr_load8(A + (size_t)m * lda + k, xv);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[m] = fmaf(xv[j], wv[j], acc[m]);
                }
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) {
            const float wv = to_float(w[k]);
#pragma unroll
            for (int m = 0; m < GR_MAX_ROWS; ++m)
                if (m < M) acc[m] = fmaf(to_float(A[(size_t)m * lda + k]), wv, acc[m]);
        }
    }
#pragma unroll
    for (int m = 0; m < GR_MAX_ROWS; ++m) {
        if (m < M) {
            const float v = warp_sum(acc[m]);
            if (lane == 0) C[(size_t)m * ldc + n] = from_float<TO>(v);
        }
    }
}

// gemm_few_batched.cu
LLMP_API int llmp_gemm_few_batched_supports(const void* A, const void* W, int M, int K, long lda, long ldw, long batch_a, long batch_w);
LLMP_API int llmp_gemm_few_batched(const void* A, const void* W, void* C, int batch, int M, int N, int K, long lda, long ldw, long ldc,
                                   long batch_a, long batch_w, long batch_c, int held, cudaStream_t stream);

// A batch of such products in one launch: product b reads A + b * batch_a and W + b * batch_w and writes C + b * batch_c
// (strides in elements; rows of any of them may lie further apart than they are long, so one product per head
// can read and write the heads of a [tokens, heads, size] tensor in place). held: 1 where W is the caller's for good, so that it may be
// read while the kernel before is still at work.
LLMP_API int llmp_gemm_simt_batched(const void* A, const void* W, void* C, int in_dtype, int out_dtype, int batch, int M, int N,
                                    int K, long lda, long ldw, long ldc, long batch_a, long batch_w, long batch_c, int held,
                                    cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    LLMP_REQUIRE(K > 0, "batched gemm: bad K %d", K);
    LLMP_REQUIRE(M <= GT_MAX_ROWS && batch <= 65535, "batched gemm: too many rows %d or products %d", M, batch);
    if (in_dtype == LLMP_BF16 && out_dtype == LLMP_BF16 && llmp_gemm_few_batched_supports(A, W, M, K, lda, ldw, batch_a, batch_w))
        return llmp_gemm_few_batched(A, W, C, batch, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, held, stream);
    if (M <= GR_MAX_ROWS && (N + 7) / 8 <= 65535) {
        dim3 rows_grid((N + 7) / 8, batch);
        const size_t esize = in_dtype == LLMP_F32 ? 4 : 2;
        const bool vec = K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && batch_a % 8 == 0 && batch_w % 8 == 0 &&
                         ((size_t)A | (size_t)W) % 16 == 0 && esize > 0;
#define LLMP_ROWS(TI, TO, WIDE)                                                                                                   \
    do {                                                                                                                          \
        llmp_launch_dependent(vec && WIDE ? gemm_rows_kernel<TI, TO, WIDE> : gemm_rows_kernel<TI, TO, false>, rows_grid, dim3(256), 0, stream,  \
                              (const TI*)A, (const TI*)W, (TO*)C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);            \
    } while (0)
        if (in_dtype == LLMP_F32 && out_dtype == LLMP_F32) LLMP_ROWS(float, float, true);
        else if (in_dtype == LLMP_BF16 && out_dtype == LLMP_BF16) LLMP_ROWS(bf16, bf16, false);
        else if (in_dtype == LLMP_BF16 && out_dtype == LLMP_F32) LLMP_ROWS(bf16, float, true);
        else {
            llmp_set_error("batched gemm: unsupported type combination in=%d out=%d", in_dtype, out_dtype);
            return 1;
        }
#undef LLMP_ROWS
        return llmp_check_launch("gemm_simt_batched (rows)");
    }
    if (!launch_nt_any(A, W, nullptr, 0, C, in_dtype, out_dtype, batch, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, stream)) {
        llmp_set_error("batched gemm: unsupported type combination in=%d out=%d", in_dtype, out_dtype);
        return 1;
    }
    return llmp_check_launch("gemm_simt_batched");
}
