// C = A * B^T on the fifth-generation tensor cores: TMA loads, tcgen05.mma with the accumulator in
// tensor memory, tcgen05.ld for the epilogue. bfloat16 operands, float32 accumulation.
//
// Both operands are K-major ([rows, K] row-major). A tile of 128 rows of A and BN rows of B is
// multiplied per block; K is walked in blocks of 64 elements (128 bytes, one swizzle span). One
// thread issues the TMA loads of a K block into a ring of STAGES shared-memory buffers (128-byte
// swizzle), one thread issues four tcgen05.mma (K = 16 each) per K block and frees the buffer with
// tcgen05.commit, four warps read the finished accumulator from tensor memory and store it.
// For the few rows of a decode step the roles are swapped: A is the weight matrix (its rows fill the
// 128-row side of the MMA), B is the activations (BN = 16, 32 or 64 rows, rows beyond M read as
// zeros by the TMA unit) and the epilogue stores the transpose; nothing is padded in memory and
// every weight byte is read once. The K order of the additions is the same for every row, so a
// row's result does not depend on the other rows of the call.
//
// Every wait on an mbarrier is bounded: when a wait runs out, the kernel records 1 in *error_flag,
// leaves its loops, frees its tensor memory and returns; the host reads the flag.
#include <cuda.h>

#include <atomic>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "tcgen05.cuh"

#define TC_THREADS 192
#define TC_BM 128
#define TC_BK 64

// BN: rows of B per tile (the N of the MMA). SWAP: store the transpose (Y[b row, a row]).
template <int BN, int STAGES, bool SWAP, typename TO>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, TO* __restrict__ Y,
               int rows_a, int rows_b, int K, long ldy, int* __restrict__ error_flag) {
    extern __shared__ unsigned char tc_raw[];
    constexpr uint32_t A_BYTES = TC_BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr uint32_t COLS = BN < 32 ? 32 : BN;               // tensor-memory columns (a power of two >= 32)
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], accum_bar;
    __shared__ uint32_t tmem_slot;

    // the swizzled tiles want 1024-byte alignment
    const uint32_t raw_addr = tc_smem_u32(tc_raw);
    unsigned char* tiles = tc_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int a0 = blockIdx.x * TC_BM, b0 = blockIdx.y * BN;
    const int kblocks = (K + TC_BK - 1) / TC_BK;

    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&accum_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // producer: TMA loads of K block kb into buffer kb % STAGES
            for (int kb = 0; kb < kblocks; ++kb) {
                const int s = kb % STAGES;
                if (kb >= STAGES && !mbar_wait(&empty_bar[s], ((kb / STAGES) - 1) & 1, error_flag)) break;
                mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                unsigned char* stage = tiles + (size_t)s * STAGE_BYTES;
                tma_load_2d(stage, &map_a, kb * TC_BK, a0, &full_bar[s]);
                tma_load_2d(stage + A_BYTES, &map_b, kb * TC_BK, b0, &full_bar[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // MMA issuer
            constexpr uint32_t idesc = umma_idesc(TC_BM, BN);
            bool ok = true;
            for (int kb = 0; kb < kblocks && ok; ++kb) {
                const int s = kb % STAGES;
                ok = mbar_wait(&full_bar[s], (kb / STAGES) & 1, error_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a_addr = tc_smem_u32(tiles + (size_t)s * STAGE_BYTES);
                const uint64_t desc_a = umma_desc(a_addr), desc_b = umma_desc(a_addr + A_BYTES);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k)     // 32 bytes along K per MMA: 2 units of 16 bytes
                    umma_f16(tmem_base, desc_a + 2 * k, desc_b + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                umma_commit(&empty_bar[s]);              // the buffer is free when these MMAs have read it
            }
            if (ok) umma_commit(&accum_bar);             // the accumulator is complete
        }
    } else {
        // epilogue: warp w reads the 32 tensor-memory lanes of its quarter (w % 4)
        const int quarter = warp & 3;
        if (mbar_wait(&accum_bar, 0, error_flag)) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int arow = a0 + quarter * 32 + lane;
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float v[16];
                tmem_ld_16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
                if (SWAP) {
                    // Y[b row, a row]: the lanes of a warp hold consecutive a rows
                    if (arow < rows_a) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (b0 + c0 + j < rows_b) Y[(size_t)(b0 + c0 + j) * ldy + arow] = from_float<TO>(v[j]);
                    }
                } else if (arow < rows_a) {
                    TO* dst = Y + (size_t)arow * ldy + b0 + c0;
                    if (b0 + c0 + 16 <= rows_b && ((size_t)dst % 16) == 0) {
                        if (sizeof(TO) == 4) {
#pragma unroll
                            for (int j = 0; j < 16; j += 4)
                                *reinterpret_cast<float4*>(reinterpret_cast<float*>(dst) + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; j += 8) {
                                uint4 pack;
                                __nv_bfloat162 h0 = __floats2bfloat162_rn(v[j], v[j + 1]), h1 = __floats2bfloat162_rn(v[j + 2], v[j + 3]);
                                __nv_bfloat162 h2 = __floats2bfloat162_rn(v[j + 4], v[j + 5]), h3 = __floats2bfloat162_rn(v[j + 6], v[j + 7]);
                                pack.x = *reinterpret_cast<unsigned*>(&h0);
                                pack.y = *reinterpret_cast<unsigned*>(&h1);
                                pack.z = *reinterpret_cast<unsigned*>(&h2);
                                pack.w = *reinterpret_cast<unsigned*>(&h3);
                                *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(dst) + j) = pack;
                            }
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (b0 + c0 + j < rows_b) dst[j] = from_float<TO>(v[j]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(COLS) : "memory");
    }
}

// ---- split-K for the few rows of a decode step ----------------------------------------------------------
// With fewer 128-row tiles of the weight matrix than SMs, one tile per block would leave most of the
// GPU without work and every working SM with more bytes to pull than it can. The blocks of a
// thread-block cluster (1, 1, splits) therefore share one output tile and each takes a contiguous
// share of the K blocks. When all of them are done, the blocks of rank 1.. write their float32
// partial tiles into the shared memory of the rank-0 block (distributed shared memory; its TMA ring
// is free by then), and rank 0 adds them in rank order and stores. No scratch in global memory, no
// atomics, and a fixed order of additions.
template <int BN, int STAGES, typename TO>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_splitk_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      TO* __restrict__ Y, int rows_a, int rows_b, int K, long ldy, int splits,
                      int* __restrict__ error_flag) {
    extern __shared__ unsigned char tc_raw[];
    constexpr uint32_t A_BYTES = TC_BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr uint32_t COLS = BN < 32 ? 32 : BN;
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], accum_bar;
    __shared__ uint32_t tmem_slot;
    const uint32_t raw_addr = tc_smem_u32(tc_raw);
    unsigned char* tiles = tc_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int a0 = blockIdx.x * TC_BM, b0 = blockIdx.y * BN;
    const int rank = (int)cluster_ctarank();
    pdl_trigger();                                   // the kernel after this one may take its places
    const int kblocks = (K + TC_BK - 1) / TC_BK;
    const int per = (kblocks + splits - 1) / splits;
    const int kb0 = rank * per;
    const int count = kb0 >= kblocks ? 0 : (kb0 + per <= kblocks ? per : kblocks - kb0);

    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&accum_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    float v[BN];                     // this thread's row of the partial tile (epilogue warps only)
    bool have = false;
    const int quarter = warp & 3;
    if (warp == 0) {
        if (lane == 0) {
            // A holds the weights: the ring is filled with them at once. B, the activations, may still be in the
            // making by the kernel before this one: its loads follow after pdl_wait().
            const int ahead = count < STAGES ? count : STAGES;
            for (int i = 0; i < ahead; ++i) {
                mbar_expect_tx(&full_bar[i], STAGE_BYTES);
                tma_load_2d(tiles + (size_t)i * STAGE_BYTES, &map_a, (kb0 + i) * TC_BK, a0, &full_bar[i]);
            }
            pdl_wait();
            for (int i = 0; i < ahead; ++i)
                tma_load_2d(tiles + (size_t)i * STAGE_BYTES + A_BYTES, &map_b, (kb0 + i) * TC_BK, b0, &full_bar[i]);
            for (int i = ahead; i < count; ++i) {
                const int s = i % STAGES;
                if (!mbar_wait(&empty_bar[s], ((i / STAGES) - 1) & 1, error_flag)) break;
                mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                unsigned char* stage = tiles + (size_t)s * STAGE_BYTES;
                tma_load_2d(stage, &map_a, (kb0 + i) * TC_BK, a0, &full_bar[s]);
                tma_load_2d(stage + A_BYTES, &map_b, (kb0 + i) * TC_BK, b0, &full_bar[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc(TC_BM, BN);
            bool ok = true;
            for (int i = 0; i < count; ++i) {
                const int s = i % STAGES;
                ok = mbar_wait(&full_bar[s], (i / STAGES) & 1, error_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a_addr = tc_smem_u32(tiles + (size_t)s * STAGE_BYTES);
                const uint64_t desc_a = umma_desc(a_addr), desc_b = umma_desc(a_addr + A_BYTES);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k)
                    umma_f16(tmem_base, desc_a + 2 * k, desc_b + 2 * k, idesc, (i | k) != 0 ? 1u : 0u);
                umma_commit(&empty_bar[s]);
            }
            if (ok && count > 0) umma_commit(&accum_bar);
        }
    } else if (count > 0) {
        if (mbar_wait(&accum_bar, 0, error_flag)) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float part[16];
                tmem_ld_16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, part);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[c0 + j] = part[j];
            }
            have = true;
        }
    }
    // every block of the cluster has finished reading its ring: rank 0's ring may now receive partial tiles
    cluster_sync_all();
    const int row = quarter * 32 + lane;                 // row of the tile held by an epilogue thread
    if (warp >= 2 && rank != 0 && have) {
        const uint32_t base = tc_smem_u32(tiles) + (uint32_t)((rank - 1) * BN * TC_BM + row) * 4u;
#pragma unroll
        for (int j = 0; j < BN; ++j) st_cluster_f32(base + (uint32_t)(j * TC_BM) * 4u, 0u, v[j]);
    }
    cluster_sync_all();
    if (warp >= 2 && rank == 0 && have) {
        const float* slots = reinterpret_cast<const float*>(tiles);
        const int arow = a0 + row;
        if (arow < rows_a) {
#pragma unroll
            for (int j = 0; j < BN; ++j) {
                float sum = v[j];
                for (int r = 1; r < splits; ++r) {
                    const int rk0 = r * per;
                    if (rk0 < kblocks) sum += slots[((size_t)(r - 1) * BN + j) * TC_BM + row];     // rank order
                }
                if (b0 + j < rows_b) Y[(size_t)(b0 + j) * ldy + arow] = from_float<TO>(sum);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(COLS) : "memory");
    }
}

// ---- persistent kernel for many rows (prompt portions) -------------------------------------------------
// One block per SM walks output tiles of 128 x BN (tile t: column block t / m_tiles, row block
// t % m_tiles, so blocks that run side by side share a weight tile through L2). The TMA ring keeps
// running across tiles. Two accumulators live in tensor memory: while the four epilogue warps read
// tile i out of one (tcgen05.ld, convert, store), the MMA thread already fills the other with tile
// i + 1. Barriers: full/empty per ring stage, accumulator-full/accumulator-empty per accumulator.
template <int BN, int STAGES, typename TO>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_persistent_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                          TO* __restrict__ Y, int rows_a, int rows_b, int K, long ldy, int* __restrict__ error_flag) {
    extern __shared__ unsigned char tc_raw[];
    constexpr uint32_t A_BYTES = TC_BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr uint32_t COLS = 2 * BN;                          // two accumulators (BN = 32, 128 or 256: a power of two)
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    const uint32_t raw_addr = tc_smem_u32(tc_raw);
    unsigned char* tiles = tc_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kblocks = (K + TC_BK - 1) / TC_BK;
    const int m_tiles = (rows_a + TC_BM - 1) / TC_BM, n_tiles = (rows_b + BN - 1) / BN;
    const int total_tiles = m_tiles * n_tiles;

    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_full[0], 1);
        mbar_init(&acc_full[1], 1);
        mbar_init(&acc_empty[0], 4);       // one arrival per epilogue warp
        mbar_init(&acc_empty[1], 4);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    pdl_wait();                                                // what the kernels before wrote is complete
    pdl_trigger();                                             // (after the allocation: nobody else's may come between)

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;                                          // K blocks issued so far, over all tiles
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const int a0 = (tile % m_tiles) * TC_BM, b0 = (tile / m_tiles) * BN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait(&empty_bar[s], ((it / STAGES) - 1) & 1, error_flag)) { ok = false; break; }
                    mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                    unsigned char* stage = tiles + (size_t)s * STAGE_BYTES;
                    tma_load_2d(stage, &map_a, kb * TC_BK, a0, &full_bar[s]);
                    tma_load_2d(stage + A_BYTES, &map_b, kb * TC_BK, b0, &full_bar[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc(TC_BM, BN);
            int it = 0, n = 0;                                   // K blocks consumed, tiles done
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++n) {
                const int acc = n & 1;
                // the epilogue must have drained this accumulator (its use n / 2 - 1)
                if (n >= 2 && !mbar_wait(&acc_empty[acc], ((n >> 1) - 1) & 1, error_flag)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t d_addr = tmem_base + (uint32_t)(acc * BN);
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(&full_bar[s], (it / STAGES) & 1, error_flag)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t a_addr = tc_smem_u32(tiles + (size_t)s * STAGE_BYTES);
                    const uint64_t desc_a = umma_desc(a_addr), desc_b = umma_desc(a_addr + A_BYTES);
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        umma_f16(d_addr, desc_a + 2 * k, desc_b + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                    umma_commit(&empty_bar[s]);
                }
                if (ok) umma_commit(&acc_full[acc]);
            }
        }
    } else {
        const int quarter = warp & 3;
        float* stage_rows = reinterpret_cast<float*>(tiles + (size_t)STAGES * STAGE_BYTES) + quarter * TC_STAGE_FLOATS;
        const bool whole_lines = (size_t)Y % 16 == 0 && ldy * sizeof(TO) % 16 == 0;
        int n = 0;
        for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++n) {
            const int acc = n & 1;
            if (!mbar_wait(&acc_full[acc], (n >> 1) & 1, error_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int a0 = (tile % m_tiles) * TC_BM, b0 = (tile / m_tiles) * BN;
            const int row0 = a0 + quarter * 32;
#pragma unroll 2
            for (int c0 = 0; c0 < BN; c0 += 32) {
                if (b0 + c0 >= rows_b) break;
                const uint32_t from = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + c0);
                float v[32];
                {
                    float part[16];
                    tmem_ld_16(from, part);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = part[j];
                    tmem_ld_16(from + 16, part);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[16 + j] = part[j];
                }
                if (whole_lines && b0 + c0 + 32 <= rows_b) {
                    tc_store_rows(v, stage_rows, lane, [&](int r) -> TO* { return row0 + r < rows_a ? Y + (size_t)(row0 + r) * ldy + b0 + c0 : nullptr; }, (TO*)nullptr);
                } else if (row0 + lane < rows_a) {
                    tc_store_own_row(v, Y + (size_t)(row0 + lane) * ldy + b0 + c0, rows_b - b0 - c0);
                }
            }
            // this warp has read its part of the accumulator: one arrival per warp frees it for the MMA thread
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem_u32(&acc_empty[acc])) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(COLS) : "memory");
    }
}

// ---- host side: tensor maps ------------------------------------------------------------------------
EncodeTiledFn llmp_tensor_map_encoder() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &status) == cudaSuccess &&
            status == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

struct MapKey {
    const void* ptr;
    long rows, k, ld;
    int box_rows;
    bool operator==(const MapKey& o) const {
        return ptr == o.ptr && rows == o.rows && k == o.k && ld == o.ld && box_rows == o.box_rows;
    }
};
struct MapKeyHash {
    size_t operator()(const MapKey& m) const {
        size_t h = (size_t)m.ptr;
        h = h * 1000003u ^ (size_t)m.rows;
        h = h * 1000003u ^ (size_t)m.k;
        h = h * 1000003u ^ (size_t)m.ld;
        return h * 1000003u ^ (size_t)m.box_rows;
    }
};

// A [rows, K] bfloat16 row-major matrix with row pitch ld, read in boxes of box_rows x 64 elements.
int llmp_matrix_tensor_map(const void* ptr, long rows, long k, long ld, int box_rows, CUtensorMap* out) {
    static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
    static std::mutex lock;
    const MapKey key{ptr, rows, k, ld, box_rows};
    std::lock_guard<std::mutex> guard(lock);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return 0;
    }
    EncodeTiledFn fn = llmp_tensor_map_encoder();
    LLMP_REQUIRE(fn != nullptr, "gemm_tc: the driver does not provide cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(bf16)};
    const cuuint32_t box[2] = {(cuuint32_t)TC_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    LLMP_REQUIRE(rc == CUDA_SUCCESS, "gemm_tc: cuTensorMapEncodeTiled failed with code %d", (int)rc);
    if (cache.size() > 4096) cache.clear();
    cache.emplace(key, *out);
    return 0;
}

template <int BN, int STAGES, bool SWAP, typename TO>
static int launch_tc(const void* A, long rows_a, long lda, const void* B, long rows_b, long ldb, TO* Y, int K, long ldy,
                     int* error_flag, cudaStream_t stream) {
    CUtensorMap map_a, map_b;
    if (llmp_matrix_tensor_map(A, rows_a, K, lda, TC_BM, &map_a) || llmp_matrix_tensor_map(B, rows_b, K, ldb, BN, &map_b)) return 1;
    constexpr size_t smem = (size_t)STAGES * (TC_BM * 128 + BN * 128) + 1024;
    auto kernel = gemm_tc_kernel<BN, STAGES, SWAP, TO>;
    LLMP_ALLOW_SMEM(kernel, smem);
    dim3 grid((unsigned)((rows_a + TC_BM - 1) / TC_BM), (unsigned)((rows_b + BN - 1) / BN));
    LLMP_REQUIRE(grid.y <= 65535, "gemm_tc: too many column tiles");
    kernel<<<grid, TC_THREADS, smem, stream>>>(map_a, map_b, Y, (int)rows_a, (int)rows_b, K, ldy, error_flag);
    return llmp_check_launch("gemm_tc");
}

// Number of K shares for an output with `tiles` 128-row tiles: the one that fills whole waves of SMs
// best, with at least 8 K blocks per share, at most 8 shares (portable cluster size) and no more
// than fit the rank-0 ring as float32 partial tiles.
static int choose_splits(int tiles, int kblocks, int bn, size_t ring_bytes) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    int best = 1;
    double best_score = -1.0;
    for (int s = 1; s <= 8; ++s) {
        if (s > 1 && (kblocks / s < 8 || (size_t)(s - 1) * bn * TC_BM * 4 > ring_bytes)) break;
        const int per = (kblocks + s - 1) / s;
        if ((s - 1) * per >= kblocks) continue;          // the last share would be empty
        const long ctas = (long)tiles * s;
        const long waves = (ctas + sms - 1) / sms;
        const double score = (double)ctas / (double)(waves * sms) - 0.01 * (s - 1);
        if (score > best_score) {
            best_score = score;
            best = s;
        }
    }
    return best;
}

template <int BN, int STAGES, typename TO>
static int launch_tc_splitk(const void* A, long rows_a, long lda, const void* B, long rows_b, long ldb, TO* Y, int K,
                            long ldy, int* error_flag, cudaStream_t stream) {
    CUtensorMap map_a, map_b;
    if (llmp_matrix_tensor_map(A, rows_a, K, lda, TC_BM, &map_a) || llmp_matrix_tensor_map(B, rows_b, K, ldb, BN, &map_b)) return 1;
    constexpr size_t ring = (size_t)STAGES * (TC_BM * 128 + BN * 128);
    constexpr size_t smem = ring + 1024;
    auto kernel = gemm_tc_splitk_kernel<BN, STAGES, TO>;
    LLMP_ALLOW_SMEM(kernel, smem);
    const int tiles = (int)((rows_a + TC_BM - 1) / TC_BM);
    const int splits = choose_splits(tiles, (K + TC_BK - 1) / TC_BK, BN, ring);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)tiles, (unsigned)((rows_b + BN - 1) / BN), (unsigned)splits);
    config.blockDim = dim3(TC_THREADS, 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)splits;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;     // see pdl_wait() in the kernel
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = llmp_pdl_enabled() ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&config, kernel, map_a, map_b, Y, (int)rows_a, (int)rows_b, K, ldy, splits,
                                               error_flag);
    if (err != cudaSuccess) {
        llmp_set_error("gemm_tc: cluster launch failed: %s", cudaGetErrorString(err));
        return 2;
    }
    return llmp_check_launch("gemm_tc_splitk");
}

template <int BN, int STAGES, typename TO>
static int launch_tc_persistent(const void* A, long rows_a, long lda, const void* B, long rows_b, long ldb, TO* Y, int K,
                                long ldy, int* error_flag, cudaStream_t stream) {
    CUtensorMap map_a, map_b;
    if (llmp_matrix_tensor_map(A, rows_a, K, lda, TC_BM, &map_a) || llmp_matrix_tensor_map(B, rows_b, K, ldb, BN, &map_b)) return 1;
    constexpr size_t smem = (size_t)STAGES * (TC_BM * 128 + BN * 128) + 1024 + 4 * TC_STAGE_FLOATS * sizeof(float);
    auto kernel = gemm_tc_persistent_kernel<BN, STAGES, TO>;
    LLMP_ALLOW_SMEM(kernel, smem);
    const int sms = llmp_sm_count();
    const long tiles = ((rows_a + TC_BM - 1) / TC_BM) * ((rows_b + BN - 1) / BN);
    const int grid = (int)(tiles < sms ? tiles : sms);
    llmp_launch_dependent(kernel, dim3(grid), dim3(TC_THREADS), smem, stream, map_a, map_b, Y, (int)rows_a, (int)rows_b, K, ldy, error_flag);
    return llmp_check_launch("gemm_tc_persistent");
}

// ---- a narrow output of many rows with a long K --------------------------------------------------------
// 2,048 rows by 160 columns are 16 tiles, and tiles of 32 columns, 80 of them, read the rows five times and each walk the whole K (22 us
// at K 4,096). Here the NARROW_SPLITS blocks of a cluster share a tile of 128 rows and all columns, each with a share of K: the rows
// are read once, and a block's ring asks for a good part of its share at once. The accumulators are put into the blocks' shared
// memory, and each block adds a share of the tile's rows from all of them, in their order. 12.6 us; 300 rows 22.1 and 11.9; 96 columns,
// K 2,048 12.8 and 7.9. Eight blocks: 9.0 for 300 rows, but 18.1 for 2,048, whose 16 clusters do not fit the SMs' groups at once; two: 19.6.
// The shares follow from K alone, so a row has the same bits among any number of rows that go this way (another number takes tiles). smem: the ring, then the same place for the accumulator, rows padded by 4 floats.
constexpr int NARROW_SPLITS = 4, NARROW_MAX_COLS = 256, NARROW_MAX_STAGES = 8;
template <typename TO>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_narrow_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, TO* __restrict__ Y, int M, int N,
                      int K, long ldy, int bn, int stages, int* __restrict__ error_flag) {
    extern __shared__ unsigned char tc_raw[];
    __shared__ __align__(8) uint64_t full_bar[NARROW_MAX_STAGES], empty_bar[NARROW_MAX_STAGES], acc_full;
    __shared__ uint32_t tmem_slot;
    const uint32_t raw_addr = tc_smem_u32(tc_raw);
    unsigned char* tiles = tc_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
    const uint32_t a_bytes = TC_BM * 128, stage_bytes = a_bytes + (uint32_t)bn * 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_ctarank(), m0 = blockIdx.x * TC_BM;
    const int kblocks = (K + TC_BK - 1) / TC_BK, per = (kblocks + NARROW_SPLITS - 1) / NARROW_SPLITS;
    const int kb0 = rank * per, count = max(0, min(kblocks, kb0 + per) - kb0);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_slot)), "r"((uint32_t)NARROW_MAX_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    pdl_wait();                                                // what the kernels before wrote is complete
    pdl_trigger();
    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (; it < count; ++it) {
                const int s = it % stages;
                if (it >= stages && !mbar_wait(&empty_bar[s], ((it / stages) - 1) & 1, error_flag)) break;
                mbar_expect_tx(&full_bar[s], stage_bytes);
                unsigned char* stage = tiles + (size_t)s * stage_bytes;
                tma_load_2d(stage, &map_a, (kb0 + it) * TC_BK, m0, &full_bar[s]);
                tma_load_2d(stage + a_bytes, &map_b, (kb0 + it) * TC_BK, 0, &full_bar[s]);
            }
            // the copies of the last stages are over before the block may end
            for (int k = it > stages ? it - stages : 0; k < it; ++k) mbar_wait(&full_bar[k % stages], (k / stages) & 1, error_flag);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0 && count > 0) {
            const uint32_t idesc = umma_idesc(TC_BM, bn);
            bool ok = true;
            for (int it = 0; it < count; ++it) {
                const int s = it % stages;
                if (!mbar_wait(&full_bar[s], (it / stages) & 1, error_flag)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a_addr = tc_smem_u32(tiles + (size_t)s * stage_bytes);
                const uint64_t desc_a = umma_desc(a_addr), desc_b = umma_desc(a_addr + a_bytes);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k) umma_f16(tmem_base, desc_a + 2 * k, desc_b + 2 * k, idesc, (it | k) != 0 ? 1u : 0u);
                umma_commit(&empty_bar[s]);
            }
            if (ok) umma_commit(&acc_full);
        }
        __syncwarp();
    }
    const int pitch = bn + 4;
    float* sums = reinterpret_cast<float*>(tiles);
    bool made = count > 0;
    if (warp >= 2 && made) {                                   // the products are done with the ring before it is written
        made = mbar_wait(&acc_full, 0, error_flag);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    }
    __syncthreads();
    if (warp >= 2) {
        const int quarter = warp & 3;
        float* row = sums + (size_t)(quarter * 32 + lane) * pitch;
        made = __all_sync(0xffffffffu, made);
        for (int c = 0; c < bn; c += 16) {
            float v[16] = {};
            if (made) tmem_ld_16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c, v);
#pragma unroll
            for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(row + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
    }
    __syncwarp();
    cluster_sync_all();
    const int quads = bn / 4;
    for (int e = threadIdx.x; e < (TC_BM / NARROW_SPLITS) * quads; e += TC_THREADS) {
        const int r = rank * (TC_BM / NARROW_SPLITS) + e / quads, c = e % quads * 4, m = m0 + r;
        if (m >= M || c >= N) continue;
        const uint32_t at = tc_smem_u32(sums + (size_t)r * pitch + c);
        float4 part[NARROW_SPLITS];
#pragma unroll
        for (int q = 0; q < NARROW_SPLITS; ++q) {
            uint32_t there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(there) : "r"(at), "r"(q));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(part[q].x), "=f"(part[q].y), "=f"(part[q].z), "=f"(part[q].w) : "r"(there) : "memory");
        }
        float4 s = part[0];
#pragma unroll
        for (int q = 1; q < NARROW_SPLITS; ++q) { s.x += part[q].x; s.y += part[q].y; s.z += part[q].z; s.w += part[q].w; }
        TO* to = Y + (size_t)m * ldy + c;
        to[0] = from_float<TO>(s.x);
        if (c + 1 < N) to[1] = from_float<TO>(s.y);
        if (c + 2 < N) to[2] = from_float<TO>(s.z);
        if (c + 3 < N) to[3] = from_float<TO>(s.w);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    cluster_sync_all();                                        // nobody leaves while another block reads its sums
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"((uint32_t)NARROW_MAX_COLS) : "memory");
    }
}

constexpr size_t NARROW_ROOM = 200 * 1024;                     // one block an SM: tensor memory is not shared with another's

template <typename TO> static cudaLaunchConfig_t narrow_config(int M, cudaLaunchAttribute (&attr)[2]) {
    auto kernel = gemm_tc_narrow_kernel<TO>;
    LLMP_ALLOW_SMEM(kernel, NARROW_ROOM + 1024);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((M + TC_BM - 1) / TC_BM, NARROW_SPLITS);
    config.blockDim = dim3(TC_THREADS);
    config.dynamicSmemBytes = NARROW_ROOM + 1024;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = NARROW_SPLITS;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = 1;
    return config;
}

// Clusters that have their places at once. A cluster lies in one group of SMs, whose number is not a multiple of its blocks everywhere: 148
// SMs hold fewer than 37 of four blocks. Asked once a device.
template <typename TO> static int narrow_clusters() {
    static std::atomic<int> known[64];
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device >= 64) return 0;
    int n = known[device].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t config = narrow_config<TO>(1, attr);
        if (cudaOccupancyMaxActiveClusters(&n, gemm_tc_narrow_kernel<TO>, &config) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = -1;
        }
        known[device].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Up to 256 columns and K of 1,024 or more, while the clusters are one round. Microseconds in tiles and in clusters, K 768, 1,024, 1,536: 2,048
// rows by 96 columns 6.4 and 5.9, 7.5 and 6.6, 9.7 and 7.5; by 160 columns 6.5 and 7.3, 7.7 and 7.8, 10.2 and 8.6; 4,096 rows by
// 256 columns of K 2,048 15.6 and 12.1, 4,736 rows, a second round of clusters, 15.8 and 21.5.
template <typename TO> static bool narrow_serves(int M, int N, int K) {
    return M > 64 && N <= NARROW_MAX_COLS && K >= 1024 && (M + TC_BM - 1) / TC_BM <= narrow_clusters<TO>();
}

template <typename TO>
static int launch_tc_narrow(const void* A, int M, long lda, const void* B, int N, long ldb, TO* Y, int K, long ldy, int* error_flag, cudaStream_t stream) {
    const int bn = (N + 15) / 16 * 16;
    CUtensorMap map_a, map_b;
    if (llmp_matrix_tensor_map(A, M, K, lda, TC_BM, &map_a) || llmp_matrix_tensor_map(B, N, K, ldb, bn, &map_b)) return 1;
    const size_t stage = TC_BM * 128 + (size_t)bn * 128;
    const int stages = NARROW_ROOM / stage < NARROW_MAX_STAGES ? (int)(NARROW_ROOM / stage) : NARROW_MAX_STAGES;
    LLMP_REQUIRE((size_t)TC_BM * (bn + 4) * sizeof(float) <= NARROW_ROOM, "gemm_tc: %d columns do not fit", N);
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t config = narrow_config<TO>(M, attr);
    config.stream = stream;
    config.numAttrs = llmp_pdl_enabled() ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&config, gemm_tc_narrow_kernel<TO>, map_a, map_b, Y, M, N, K, ldy, bn, stages, error_flag);
    if (err != cudaSuccess) {
        llmp_set_error("gemm_tc: cluster launch failed: %s", cudaGetErrorString(err));
        return 2;
    }
    return llmp_check_launch("gemm_tc_narrow");
}

template <typename TO>
static int dispatch_tc(const void* X, const void* W, TO* Y, int M, int N, int K, long ldx, long ldw, long ldy,
                       int* error_flag, cudaStream_t stream) {
    if (M <= 16) return launch_tc_splitk<16, 10, TO>(W, N, ldw, X, M, ldx, Y, K, ldy, error_flag, stream);
    if (M <= 32) return launch_tc_splitk<32, 9, TO>(W, N, ldw, X, M, ldx, Y, K, ldy, error_flag, stream);
    if (M <= 64) return launch_tc_splitk<64, 8, TO>(W, N, ldw, X, M, ldx, Y, K, ldy, error_flag, stream);
    if (narrow_serves<TO>(M, N, K)) return launch_tc_narrow(X, M, ldx, W, N, ldw, Y, K, ldy, error_flag, stream);
    // 128 x 256 tiles do twice the work per byte read from shared memory; 128 x 128 only for narrow outputs, and 128 x 32 where the SMs
    // take even those in one go: 2,048 rows, 160 columns, K 4,096 26.2 us -> 22.2; 96 columns, K 2,048 15.8 -> 12.6. (Sharing K among
    // the blocks of a cluster, 64 rows by 128 columns each, lost: 31 and 25 us; for a long K the kernel above.)
    if (N < 256 && (long)((M + TC_BM - 1) / TC_BM) * ((N + 31) / 32) <= llmp_sm_count())
        return launch_tc_persistent<32, 8, TO>(X, M, ldx, W, N, ldw, Y, K, ldy, error_flag, stream);
    if (N >= 256) return launch_tc_persistent<256, 4, TO>(X, M, ldx, W, N, ldw, Y, K, ldy, error_flag, stream);
    return launch_tc_persistent<128, 6, TO>(X, M, ldx, W, N, ldw, Y, K, ldy, error_flag, stream);
}

// Y[M, N] = X[M, K] * W[N, K]^T, bfloat16 operands with 16-byte aligned rows (K, ldx, ldw multiples of 8),
// Y bfloat16 or float32. error_flag: one int in device memory that the kernel sets to 1 when a wait
// ran out (the host checks it after synchronising).
// Whether a product of these sizes is shared in clusters.
LLMP_API int llmp_gemm_tc_narrow_serves(int out_dtype, int M, int N, int K) {
    return out_dtype == LLMP_F32 ? narrow_serves<float>(M, N, K) : narrow_serves<bf16>(M, N, K);
}

LLMP_API int llmp_gemm_tc(const void* X, const void* W, void* Y, int out_dtype, int M, int N, int K, long ldx, long ldw,
                          long ldy, int* error_flag, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    LLMP_REQUIRE(K > 0 && K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0,
                 "gemm_tc: K=%d and the row strides (%ld, %ld) must be multiples of 8", K, ldx, ldw);
    LLMP_REQUIRE(((size_t)X % 16) == 0 && ((size_t)W % 16) == 0, "gemm_tc: operands must be 16-byte aligned");
    LLMP_REQUIRE(error_flag != nullptr, "gemm_tc: an error flag in device memory is required");
    if (out_dtype == LLMP_F32) return dispatch_tc<float>(X, W, (float*)Y, M, N, K, ldx, ldw, ldy, error_flag, stream);
    return dispatch_tc<bf16>(X, W, (bf16*)Y, M, N, K, ldx, ldw, ldy, error_flag, stream);
}
