// Latent attention of long prompt portions with the heads' keys and values formed (bfloat16, fifth-generation tensor cores).
//
// The rows of the cache are latents that all heads share. Few new rows attend over them as they are (latent_attention_mma.cu):
// the maps of keys and values move to the query's side, and a (query, key, head) costs 2 rank + rot multiply-adds. For many new
// rows that is the dear order: with the keys W_uk c and values W_uv c formed once per key (one product over the rows of the
// request, as large as the two maps it replaces), a (query, key, head) costs dim + rot + vdim. At rank 512, rot 64 and heads of 128
// that is 320 against 1,088: 2,048 tokens of 16 heads took 627 us there (121 TFLOP/s of the larger count) beside 28 us of maps.
//
// latent_gather: the cached rows of every request, page by page, become one matrix with each request's rows padded to whole key
// tiles by zeros. The caller multiplies it by [W_uk; W_uv]. latent_prompt_kernel: a block takes 128 new tokens of a request and one
// head, with the roles and the softmax of attention_prefill_tc.cu: S = Q K^T with Q and K in planes of 64 columns (the last one
// the rotated part, whose keys all heads share and which stays in the gathered rows), P over S in tensor memory, O += P V with V
// as an MN-major operand. A key tile has as many keys as leave two blocks room on an SM (96 with heads of 128 + 64, 128 with 64 +
// 32), so that one's products run under the other's softmax.
//
// Every wait on an mbarrier is bounded (mbar_wait): when one runs out the kernel records it in *error_flag and goes on.
#include "common.cuh"
#include "prefill_tc.cuh"

namespace {

constexpr int LP_ROWS = 128;
constexpr int LP_THREADS = 192;                          // four softmax warps, one load warp, one MMA warp
constexpr int LP_Q_PLANE = LP_ROWS * 128;                // bytes of 128 rows of 64 entries
constexpr int LP_TMEM_COLS = 256, LP_TMEM_O = 128;       // S (up to 128 columns) and O

struct PromptParams {
    const bf16* q; long q_t, q_h;                        // [tokens][heads][dim + rot]
    bf16* out; long o_t, o_h;                            // [tokens][heads][vdim]
    const int* q_start; const int* ctx_len;
    const int* tile_req; const int* tile_tok0; const int* tile_base;    // base: the request's first row of the gathered matrix
    const float* sink;                                   // [heads] or null
    int H, rot, rank, num_tiles, num_sms;
    float scale;
    int* error_flag;
};

// An eighth of a key tile of the gathered matrix a block: its rows from the pages, zeros past the request's keys.
constexpr int LG_SHARES = 8;
__global__ void __launch_bounds__(256) latent_gather_kernel(const bf16* __restrict__ pages, const int* __restrict__ tables, int table_stride,
                                                            const int* __restrict__ ctx_len, const int* __restrict__ block_req,
                                                            const int* __restrict__ block_key0, int keys, int page_size, int dk,
                                                            bf16* __restrict__ rows) {
    const int r = block_req[blockIdx.x], ctx = ctx_len[r], pieces = dk / 8;
    const int own = keys / LG_SHARES, row0 = blockIdx.y * own, key0 = block_key0[blockIdx.x] + row0;
    rows += ((size_t)blockIdx.x * keys + row0) * dk;
    for (int i = threadIdx.x; i < own * pieces; i += blockDim.x) {
        const int key = key0 + i / pieces, e = i % pieces * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (key < ctx) {
            const int page = tables[(size_t)r * table_stride + key / page_size];
            if (page >= 0) v = *reinterpret_cast<const uint4*>(pages + ((size_t)page * page_size + key % page_size) * dk + e);
        }
        *reinterpret_cast<uint4*>(rows + (size_t)(i / pieces) * dk + e) = v;
    }
}

// Shared-memory descriptor of an MN-major operand in the 128-byte swizzle: rows of 64 contiguous entries of the MN dimension, one
// row per K index, groups of 8 K indices 1024 bytes apart, the next 64 entries `plane` bytes further.
__device__ __forceinline__ uint64_t lp_desc_mn_major(uint32_t smem_addr, uint32_t plane) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(plane >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// DP planes of 64 unrotated query and key entries, VP planes of 64 value entries, KEYS keys a tile.
template <int DP, int VP, int KEYS>
__global__ void __launch_bounds__(LP_THREADS, 2)
latent_prompt_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_rows, const PromptParams p) {
    extern __shared__ unsigned char lp_raw[];
    __shared__ __align__(8) uint64_t k_full, v_full, s_done, o_done, p_ready;
    __shared__ uint32_t tmem_slot;
    constexpr int QP = DP + 1, PLANE = KEYS * 128, CHUNKS = KEYS / 32;
    const uint32_t raw_addr = tc_smem_u32(lp_raw);
    unsigned char* Qs = lp_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);   // [QP][128 rows][128 bytes]
    unsigned char* Ks = Qs + QP * LP_Q_PLANE;                                  // [QP][KEYS][128 bytes]
    unsigned char* Vs = Ks + QP * PLANE;                                       // [VP][KEYS][128 bytes]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // later tiles of a prompt see more keys: the heads of the last tile start first
    const int tile = p.num_tiles - 1 - (int)(blockIdx.x / (unsigned)p.H);
    const int h = (int)(blockIdx.x % (unsigned)p.H);
    const int r = p.tile_req[tile], tok0 = p.tile_tok0[tile], base = p.tile_base[tile];
    const int q_begin = p.q_start[r];
    const int q_len = p.q_start[r + 1] - q_begin;
    const int first_pos = p.ctx_len[r] - q_len + tok0;                         // of the tile's first token
    const int ntok = min(q_len - tok0, LP_ROWS);
    const int num_key_tiles = (first_pos + ntok - 1) / KEYS + 1;
    const int rot = p.rot;

    auto load_tile = [&](int j) {                                              // one thread of warp 4
        const int row = base + j * KEYS;
        if (j > 0) mbar_wait(&s_done, (uint32_t)((j - 1) & 1), p.error_flag);  // K is free when S of the tile before is done
        mbar_expect_tx(&k_full, QP * PLANE);
#pragma unroll
        for (int c = 0; c < DP; ++c) tma_load_2d(Ks + c * PLANE, &map_kv, (h * DP + c) * 64, row, &k_full);
        tma_load_2d(Ks + DP * PLANE, &map_rows, p.rank, row, &k_full);         // past rot: the row's end, which arrives as zeros
        if (j > 0) mbar_wait(&o_done, (uint32_t)((j - 1) & 1), p.error_flag);  // V when its P V is
        mbar_expect_tx(&v_full, VP * PLANE);
#pragma unroll
        for (int c = 0; c < VP; ++c) tma_load_2d(Vs + c * PLANE, &map_kv, (p.H * DP + h * VP + c) * 64, row, &v_full);
    };

    if (warp == 4) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_kv) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_rows) : "memory");
            mbar_init(&k_full, 1);
            mbar_init(&v_full, 1);
            mbar_init(&s_done, 1);
            mbar_init(&o_done, 1);
            mbar_init(&p_ready, LP_ROWS);
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
            load_tile(0);
        }
    } else if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_slot)), "r"(LP_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    } else {
        // Query rows in the layout of a K-major operand: 16-byte piece c of a row at place (c % 8) ^ (row % 8) of the row's
        // 128-byte line in plane c / 8; the rotated part begins a plane, and what it leaves of it is zero.
        constexpr int PIECES = QP * 8;
        const int have = DP * 8 + rot / 8;
        for (int i0 = 0; i0 < PIECES; i0 += 8) {
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = tid + (i0 + i) * 128, row = e / PIECES, c = e % PIECES;
                v[i] = make_uint4(0u, 0u, 0u, 0u);
                if (row < ntok && c < have)
                    v[i] = *reinterpret_cast<const uint4*>(p.q + (size_t)(q_begin + tok0 + row) * p.q_t + (size_t)h * p.q_h + c * 8);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = tid + (i0 + i) * 128, row = e / PIECES, c = e % PIECES;
                *reinterpret_cast<uint4*>(Qs + (c >> 3) * LP_Q_PLANE + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = v[i];
            }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    fa_fence_before();
    __syncthreads();
    fa_fence_after();
    const uint32_t tmem_base = tmem_slot;
    const uint32_t tmem_s = tmem_base, tmem_o = tmem_base + LP_TMEM_O;

    if (warp == 4) {
        if (lane == 0)
            for (int j = 1; j < num_key_tiles; ++j) load_tile(j);
    } else if (warp == 5) {
        if (lane == 0) {
            constexpr uint32_t idesc_s = umma_idesc(LP_ROWS, KEYS);
            constexpr uint32_t idesc_o = umma_idesc(LP_ROWS, VP * 64) | (1u << 16);      // B is MN-major
            const uint32_t q_addr = tc_smem_u32(Qs), k_addr = tc_smem_u32(Ks), v_addr = tc_smem_u32(Vs);
            const int steps = DP * 4 + rot / 16;
            if ((blockIdx.x / p.num_sms) & 1) __nanosleep(FA_STAGGER_NS);      // out of step with the SM's other block
            for (int j = 0; j < num_key_tiles; ++j) {
                const uint32_t parity = (uint32_t)(j & 1);
                if (j == 0) mbar_wait(&k_full, 0, p.error_flag);
                fa_fence_after();
                for (int k = 0; k < steps; ++k) {
                    const uint32_t plane = (uint32_t)(k >> 2), in = (uint32_t)(k & 3) * 32;
                    umma_f16(tmem_s, umma_desc(q_addr + plane * LP_Q_PLANE + in), umma_desc(k_addr + plane * PLANE + in), idesc_s, k != 0 ? 1u : 0u);
                }
                umma_commit(&s_done);
                mbar_wait(&v_full, parity, p.error_flag);
                if (j + 1 < num_key_tiles) mbar_wait(&k_full, parity ^ 1u, p.error_flag);
                mbar_wait(&p_ready, parity, p.error_flag);
                fa_fence_after();
#pragma unroll
                for (int k = 0; k < KEYS / 16; ++k)                            // 16 keys per MMA: 8 columns of P, 2 KB of every plane of V
                    fa_umma_a_tmem(tmem_o, tmem_s + (uint32_t)k * 8, lp_desc_mn_major(v_addr + (uint32_t)k * 2048, PLANE), idesc_o, (j | k) != 0 ? 1u : 0u);
                umma_commit(&o_done);
            }
        }
    } else {
        const uint32_t lane_field = (uint32_t)(warp * 32) << 16;              // this warp's quarter of the lanes
        const int my_pos = tid < ntok ? first_pos + tid : -1;                  // -1: the row does not exist
        const float scale_log2 = p.scale * 1.4426950408889634f;
        float m_used = -INFINITY, l_run = 0.f;
        uint32_t v[2][32];
        for (int j = 0; j < num_key_tiles; ++j) {
            const int j0 = j * KEYS;
            const bool need_mask = j0 + KEYS - 1 > first_pos;
            mbar_wait(&s_done, (uint32_t)(j & 1), p.error_flag);               // also: P V of the tile before is done
            fa_fence_after();
            // pass 1: the row's maximum, the next 32 columns in flight while 32 are reduced (the last load: pass 2's first columns)
            float mx = -INFINITY;
            FA_TMEM_LD32(tmem_s + lane_field, v[0], 0);
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                fa_tmem_wait_ld();
                FA_TMEM_LD32(tmem_s + lane_field + (c + 1) % CHUNKS * 32, v[(c + 1) & 1], 0);
                if (need_mask) fa_mask32(v[c & 1], j0 + c * 32, my_pos, 0);
                mx = fa_max32(v[c & 1], mx);
            }
            const float m_tile = mx * scale_log2;
            const bool raise = m_tile > m_used + FA_RESCALE_STEP;
            float alpha = 1.f;
            if (raise) {
                alpha = fa_ex2(m_used - m_tile);
                m_used = m_tile;
                l_run *= alpha;
            }
            fa_tmem_wait_ld();
            if (j > 0 && __any_sync(0xffffffffu, raise)) {                     // O holds the sum of the tiles before
                uint32_t (&b)[32] = v[(CHUNKS + 1) & 1];
#pragma unroll
                for (int c = 0; c < VP * 64; c += 32) {
                    FA_TMEM_LD32(tmem_o + lane_field + c, b, 0);
                    fa_tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) b[i] = __float_as_uint(__uint_as_float(b[i]) * alpha);
                    FA_TMEM_ST32(tmem_o + lane_field + c, b, 0);
                }
            }
            // pass 2: probabilities as bfloat16 pairs over the first half of S's columns (16 columns per 32 scores: always columns
            // that were read before)
            const float m_eff = m_used > -INFINITY ? m_used : 0.f;
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                uint32_t (&cur)[32] = v[(CHUNKS + c) & 1];
                uint32_t pk[16];
                if (c > 0) fa_tmem_wait_ld();
                if (c + 1 < CHUNKS) FA_TMEM_LD32(tmem_s + lane_field + (c + 1) * 32, v[(CHUNKS + c + 1) & 1], 0);
                if (need_mask) fa_mask32(cur, j0 + c * 32, my_pos, 0);
                sum += fa_exp32(cur, pk, scale_log2, m_eff);
                FA_TMEM_ST16(tmem_s + lane_field + c * 16, pk);
            }
            l_run += sum;
            fa_tmem_wait_st();
            fa_fence_before();
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem_u32(&p_ready)) : "memory");
        }
        mbar_wait(&o_done, (uint32_t)((num_key_tiles - 1) & 1), p.error_flag);
        fa_fence_after();
        float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        if (p.sink) {                                                          // a key of score sink[h] without a value
            const float sk = p.sink[h] * 1.4426950408889634f;
            const float m = fmaxf(m_used, sk);
            const float w = m_used > -INFINITY ? fa_ex2(m_used - m) : 0.f;
            inv = w / (l_run * w + fa_ex2(sk - m));
        }
        bf16* dst = p.out + (size_t)(q_begin + tok0 + (my_pos >= 0 ? tid : 0)) * p.o_t + (size_t)h * p.o_h;
#pragma unroll
        for (int c = 0; c < VP * 64; c += 32) {
            FA_TMEM_LD32(tmem_o + lane_field + c, v[0], 0);
            fa_tmem_wait_ld();
            if (my_pos >= 0) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    uint4 pack;
                    pack.x = fa_pack(__uint_as_float(v[0][i]) * inv, __uint_as_float(v[0][i + 1]) * inv);
                    pack.y = fa_pack(__uint_as_float(v[0][i + 2]) * inv, __uint_as_float(v[0][i + 3]) * inv);
                    pack.z = fa_pack(__uint_as_float(v[0][i + 4]) * inv, __uint_as_float(v[0][i + 5]) * inv);
                    pack.w = fa_pack(__uint_as_float(v[0][i + 6]) * inv, __uint_as_float(v[0][i + 7]) * inv);
                    *reinterpret_cast<uint4*>(dst + c + i) = pack;
                }
            }
        }
    }
    fa_fence_before();
    __syncthreads();
    if (warp == 5) {
        fa_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(LP_TMEM_COLS) : "memory");
    }
}

template <int DP, int VP, int KEYS>
int launch_prompt(const CUtensorMap& map_kv, const CUtensorMap& map_rows, const PromptParams& p, cudaStream_t stream) {
    constexpr size_t smem = (size_t)(DP + 1) * LP_Q_PLANE + (size_t)(DP + 1 + VP) * KEYS * 128 + 1024;
    static_assert(2 * (smem + 1024) <= 227 * 1024, "two blocks share an SM");
    LLMP_ALLOW_SMEM((latent_prompt_kernel<DP, VP, KEYS>), smem);
    latent_prompt_kernel<DP, VP, KEYS><<<(unsigned)((long)p.num_tiles * p.H), LP_THREADS, smem, stream>>>(map_kv, map_rows, p);
    return llmp_check_launch("latent_prompt_attention");
}

}  // namespace

// Keys of a key tile for heads of these sizes (the unit in which a request's gathered rows are padded); 0: not served.
LLMP_API int llmp_latent_prompt_keys(int dim, int rot, int vdim, int rank) {
    if (rot < 16 || rot > 64 || rot % 16 || rank % 64 || rank < 64) return 0;
    if (dim == 128 && vdim == 128) return 96;
    if (dim == 64 && vdim == 64) return 128;
    return 0;
}

LLMP_API int llmp_latent_gather(const void* pages, const int* tables, int table_stride, const int* ctx_len, const int* block_req,
                                const int* block_key0, int blocks, int keys, int page_size, int dk, void* rows, cudaStream_t stream) {
    if (blocks <= 0) return 0;
    LLMP_REQUIRE(keys > 0 && keys % LG_SHARES == 0 && page_size > 0 && dk % 8 == 0 && ((size_t)pages | (size_t)rows) % 16 == 0, "latent_gather: rows of %d entries", dk);
    latent_gather_kernel<<<dim3(blocks, LG_SHARES), 256, 0, stream>>>((const bf16*)pages, tables, table_stride, ctx_len, block_req, block_key0, keys, page_size, dk,
                                                     (bf16*)rows);
    return llmp_check_launch("latent_gather");
}

// kv: [rows][H dim | H vdim], the gathered rows' keys and values; rows: [rows][rank + rot]; both with the rows of a request padded to
// whole key tiles.
LLMP_API int llmp_latent_prompt_attention(const void* q, long q_t, long q_h, const void* kv, const void* rows, int num_rows, const int* q_start,
                                          const int* ctx_len, const int* tile_req, const int* tile_tok0, const int* tile_base, int num_tiles,
                                          void* out, long o_t, long o_h, int H, int dim, int rot, int vdim, int rank, float scale,
                                          const float* sink, int* error_flag, cudaStream_t stream) {
    if (num_tiles <= 0 || num_rows <= 0) return 0;
    const int keys = llmp_latent_prompt_keys(dim, rot, vdim, rank);
    LLMP_REQUIRE(keys > 0 && H > 0, "latent_prompt_attention: heads of %d + %d and %d over latents of %d are not served", dim, rot, vdim, rank);
    LLMP_REQUIRE(q_t % 8 == 0 && q_h % 8 == 0 && o_t % 8 == 0 && o_h % 8 == 0 && ((size_t)q | (size_t)out | (size_t)kv | (size_t)rows) % 16 == 0 &&
                 (rank + rot) % 8 == 0, "latent_prompt_attention: rows must be 16-byte aligned");
    LLMP_REQUIRE(num_rows % keys == 0 && (long)num_tiles * H < (1L << 31), "latent_prompt_attention: %d rows, %d tiles", num_rows, num_tiles);
    LLMP_REQUIRE(error_flag != nullptr, "latent_prompt_attention: an error flag in device memory is required");
    const long width = (long)H * (dim + vdim);
    CUtensorMap map_kv, map_rows;
    if (llmp_matrix_tensor_map(kv, num_rows, width, width, keys, &map_kv) ||
        llmp_matrix_tensor_map(rows, num_rows, rank + rot, rank + rot, keys, &map_rows)) return 1;
    PromptParams p;
    p.q = (const bf16*)q; p.q_t = q_t; p.q_h = q_h; p.out = (bf16*)out; p.o_t = o_t; p.o_h = o_h; p.q_start = q_start; p.ctx_len = ctx_len;
    p.tile_req = tile_req; p.tile_tok0 = tile_tok0; p.tile_base = tile_base; p.sink = sink; p.H = H; p.rot = rot; p.rank = rank;
    p.num_tiles = num_tiles; p.num_sms = llmp_sm_count(); p.scale = scale; p.error_flag = error_flag;
    if (dim == 128) return launch_prompt<2, 2, 96>(map_kv, map_rows, p, stream);
    return launch_prompt<1, 1, 128>(map_kv, map_rows, p, stream);
}
