// What the tcgen05 attention kernels of prompt portions share (attention_prefill_tc.cu, latent_prompt_tc.cu): products whose A
// operand lies in tensor memory, tensor-memory loads and stores of 32 columns, and the softmax's passes over them.
#pragma once
#include "tcgen05.cuh"

#define FA_RESCALE_STEP 8.0f      // in log2 units: how far a row's maximum may pass the one its sums are scaled by
#define FA_STAGGER_NS 1000        // by how much the second block of an SM starts later

// D[tmem] (+)= A[tmem] * B[smem]: the A operand is read from tensor memory (bfloat16 pairs per 32-bit column).
__device__ __forceinline__ void fa_umma_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t accumulate) {
    const uint32_t zero = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(zero) : "memory");
}

// 32 consecutive 32-bit columns of this thread's tensor-memory lane into r[OFF .. OFF + 31] (no wait).
#define FA_TMEM_LD32(taddr, r, OFF)                                                                                     \
    asm volatile(                                                                                                       \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, " \
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"                      \
        : "=r"(r[OFF + 0]), "=r"(r[OFF + 1]), "=r"(r[OFF + 2]), "=r"(r[OFF + 3]), "=r"(r[OFF + 4]), "=r"(r[OFF + 5]),   \
          "=r"(r[OFF + 6]), "=r"(r[OFF + 7]), "=r"(r[OFF + 8]), "=r"(r[OFF + 9]), "=r"(r[OFF + 10]), "=r"(r[OFF + 11]), \
          "=r"(r[OFF + 12]), "=r"(r[OFF + 13]), "=r"(r[OFF + 14]), "=r"(r[OFF + 15]), "=r"(r[OFF + 16]),                \
          "=r"(r[OFF + 17]), "=r"(r[OFF + 18]), "=r"(r[OFF + 19]), "=r"(r[OFF + 20]), "=r"(r[OFF + 21]),                \
          "=r"(r[OFF + 22]), "=r"(r[OFF + 23]), "=r"(r[OFF + 24]), "=r"(r[OFF + 25]), "=r"(r[OFF + 26]),                \
          "=r"(r[OFF + 27]), "=r"(r[OFF + 28]), "=r"(r[OFF + 29]), "=r"(r[OFF + 30]), "=r"(r[OFF + 31])                 \
        : "r"(taddr))

// r[OFF .. OFF + 31] into 32 consecutive 32-bit columns of this thread's tensor-memory lane (no wait).
#define FA_TMEM_ST32(taddr, r, OFF)                                                                                     \
    asm volatile(                                                                                                       \
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, " \
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};\n"                        \
        ::"r"(r[OFF + 0]), "r"(r[OFF + 1]), "r"(r[OFF + 2]), "r"(r[OFF + 3]), "r"(r[OFF + 4]), "r"(r[OFF + 5]),          \
          "r"(r[OFF + 6]), "r"(r[OFF + 7]), "r"(r[OFF + 8]), "r"(r[OFF + 9]), "r"(r[OFF + 10]), "r"(r[OFF + 11]),        \
          "r"(r[OFF + 12]), "r"(r[OFF + 13]), "r"(r[OFF + 14]), "r"(r[OFF + 15]), "r"(r[OFF + 16]), "r"(r[OFF + 17]),    \
          "r"(r[OFF + 18]), "r"(r[OFF + 19]), "r"(r[OFF + 20]), "r"(r[OFF + 21]), "r"(r[OFF + 22]), "r"(r[OFF + 23]),    \
          "r"(r[OFF + 24]), "r"(r[OFF + 25]), "r"(r[OFF + 26]), "r"(r[OFF + 27]), "r"(r[OFF + 28]), "r"(r[OFF + 29]),    \
          "r"(r[OFF + 30]), "r"(r[OFF + 31]), "r"(taddr)                                                                \
        : "memory")

__device__ __forceinline__ void fa_tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void fa_tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void fa_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fa_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// 2^x by the special-function unit (relative error about 2^-22; the probabilities are rounded to bfloat16 anyway)
__device__ __forceinline__ float fa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint32_t fa_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Applies the causal and window mask of one row to 32 scores that start at key `key0`.
__device__ __forceinline__ void fa_mask32(uint32_t (&v)[32], int key0, int last_ok, int first_ok) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int key = key0 + i;
        if (key > last_ok || key < first_ok) v[i] = 0xff800000u;           // -inf
    }
}

__device__ __forceinline__ float fa_max32(const uint32_t (&v)[32], float mx) {
    float m0 = mx, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;          // four chains: no serial dependency
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        m0 = fmaxf(m0, __uint_as_float(v[i]));
        m1 = fmaxf(m1, __uint_as_float(v[i + 1]));
        m2 = fmaxf(m2, __uint_as_float(v[i + 2]));
        m3 = fmaxf(m3, __uint_as_float(v[i + 3]));
    }
    return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
}

// 32 scores -> 16 packed bfloat16 pairs of 2^(s * scale - m); returns their float32 sum.
__device__ __forceinline__ float fa_exp32(const uint32_t (&v)[32], uint32_t (&pk)[16], float scale_log2, float m_eff) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float p0 = fa_ex2(fmaf(__uint_as_float(v[i]), scale_log2, -m_eff));
        const float p1 = fa_ex2(fmaf(__uint_as_float(v[i + 1]), scale_log2, -m_eff));
        s0 += p0;
        s1 += p1;
        pk[i >> 1] = fa_pack(p0, p1);
    }
    return s0 + s1;
}

#define FA_TMEM_ST16(taddr, r)                                                                                          \
    asm volatile(                                                                                                       \
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, " \
        "%15};\n"                                                                                                        \
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),  \
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)                            \
        : "memory")
