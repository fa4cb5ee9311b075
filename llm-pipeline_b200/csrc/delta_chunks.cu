// The gated delta rule of delta_rule.cu for the many tokens of a prompt portion (bfloat16 path), in chunks of 16 tokens.
//
//   S <- diag(g_t) S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
// Token by token that is a chain of dependent passes over the state, 0.3 us each whatever its size. Within a chunk, with G_t the
// product of the chunk's decays up to t (per channel) and S the state before the chunk, the u are the solution of a triangular
// system that does not depend on S but for its right-hand side:
//   A[t, j] = sum_c k_t k_j G_t / G_j (j < t),   T = (I + diag(beta) A)^-1 diag(beta),   U = T V - (T (G k)) S
//   o_t = (G_t q_t)^T S + sum_(j <= t) B[t, j] u_j,   B[t, j] = sum_c q_t k_j G_t / G_j
//   S' = diag(G_16) S + sum_j (G_16 / G_j k_j) u_j^T
// Two launches:
//   1. every (chunk, head) side by side: unit vectors, decays and beta from the projections (the work of delta_prep), A, B, T, and
//      what the chain needs of a chunk: W = T (G k), Q = G q, K = G_16 / G k, B, Y = T V, G_16;
//   2. the chain: a block per (request, head, 16 value columns) walks the request's chunks with the state in registers: four
//      products of 16 tokens a chunk on the tensor cores instead of 16 passes.
// Everything is float32; ratios of decays are products of the decays between (never above one, so nothing overflows however fast a
// channel forgets; exponentials of differences of summed logarithms lose a slow decay's bits to a fast one before it: 5e-3 of the
// state after a reset). Where a float32 number enters a product it is split into three bfloat16 pieces, which hold all of
// its 24 bits, and of the nine products of pieces the six larger are summed in float32, the largest apart: outputs and state are
// as far from 64 bits as token by token (1.2e-7 to 3e-7 at decays from fast to slow, and after resets; with two pieces and three
// products 5e-6, at 47 us less). The operands of launch 2 lie in scratch in the order of its fragments, pieces beside each other,
// and are copied as they are. A layer of 2,048 tokens and 16 heads of 128 x 128 takes 358 us, 809 token by token. Launch 1 (96 us
// with cold caches) is issue-bound at 44 % with 14 warps an SM; launch 2 (148) is the chain's latency, 1.16 us a chunk (tensor pipe
// 32 %, a warp a scheduler). On the way: 32 columns a block with fragments loaded from global memory,
// two barriers a chunk (each slower by 15 to 45 %).
#include "tcgen05.cuh"

namespace {

constexpr int DC_TOKENS = 16;             // tokens of a chunk
constexpr int DC_PREP_THREADS = 128;
constexpr int DC_CHAIN_THREADS = 128;     // of the chain: four quarters of the channels
constexpr int DC_STAGES = 4;              // records of its ring

struct DeltaChunkArgs {
    const float* q; long q_t; const float* k; long k_t; const float* v; long v_t;     // as the convolution left them
    const float* decay; long decay_t; const float* beta; long beta_t;                 // pre-activations
    const float* a_log; const float* dt_bias;                                         // [H], [H d]
    float* state; long state_slot; long state_half;                                   // copy: [H][d][dv]
    const int* q_start; const int* slots; const int* positions;
    float* o; long o_t;
    unsigned char* scratch;               // [chunks][H] records
    int* error_flag;
    const int* list;                      // the requests to take, ascending; null: all
    int requests, H, G, dv;
};

// Bytes of a record, whose parts are, in order: W, Q, K (96 a channel each), B (1536), Y (64 a column), G (4 a channel).
__host__ __device__ constexpr int dc_record(int d, int dv) { return 3 * d * 96 + 1536 + dv * 64 + d * 4; }

__device__ __forceinline__ float dc_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

__device__ __forceinline__ void dc_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// A float as three bfloat16 numbers that add up to it.
__device__ __forceinline__ void dc_split(float u, bf16& hi, bf16& mid, bf16& lo) {
    hi = __float2bfloat16_rn(u);
    const float rest = u - __bfloat162float(hi);
    mid = __float2bfloat16_rn(rest);
    lo = __float2bfloat16_rn(rest - __bfloat162float(mid));
}
// Two floats as three such pairs.
__device__ __forceinline__ void dc_split(float u, float v, unsigned& hi, unsigned& mid, unsigned& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(u, v);
    const float ru = u - __low2float(h), rv = v - __high2float(h);
    const __nv_bfloat162 m = __floats2bfloat162_rn(ru, rv);
    const __nv_bfloat162 l = __floats2bfloat162_rn(ru - __low2float(m), rv - __high2float(m));
    hi = *reinterpret_cast<const unsigned*>(&h);
    mid = *reinterpret_cast<const unsigned*>(&m);
    lo = *reinterpret_cast<const unsigned*>(&l);
}
// A fragment of a record (a k16 x n8 operand, split): the larger two pieces of a lane's two words beside each other, then all
// lanes' smallest.
constexpr int DC_FRAGMENT = 768;
struct DcFragment { unsigned piece[3][2]; };
__device__ __forceinline__ DcFragment dc_fragment(const unsigned char* at, int lane) {
    const uint4 a = *reinterpret_cast<const uint4*>(at + lane * 16);
    const uint2 b = *reinterpret_cast<const uint2*>(at + 512 + lane * 8);
    return {{{a.x, a.y}, {a.z, a.w}, {b.x, b.y}}};
}
__device__ __forceinline__ void dc_put(unsigned char* at, int lane, const unsigned (&b0)[3], const unsigned (&b1)[3]) {
    *reinterpret_cast<uint4*>(at + lane * 16) = make_uint4(b0[0], b1[0], b0[1], b1[1]);
    *reinterpret_cast<uint2*>(at + 512 + lane * 8) = make_uint2(b0[2], b1[2]);
}
// one entry of a fragment: of a lane's word `word` the half `half`
__device__ __forceinline__ void dc_put(unsigned char* at, int lane, int word, int half, float x) {
    bf16* pair = reinterpret_cast<bf16*>(at + lane * 16 + word * 4) + half;
    dc_split(x, pair[0], pair[4], reinterpret_cast<bf16*>(at + 512 + lane * 8 + word * 4)[half]);
}
// Products of split factors with T operands: of the nine products of pieces the six larger ones, the largest apart from the others,
// so that neither loses bits to the other's rounding.
template <int T> __device__ __forceinline__ void dc_products(float (&big)[T][4], float (&small)[T][4], const unsigned (&a)[3][4], const DcFragment (&b)[T]) {
    constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int n = 0; n < T; ++n) dc_mma(i == 5 ? big[n] : small[n], a[PA[i]], b[n].piece[PB[i]][0], b[n].piece[PB[i]][1]);
}
__device__ __forceinline__ float dc_dot(const float4& a, const float4& b, float s) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s))));
}
// The sums over 16 neighbouring lanes of v[0] .. v[15]: lane i of them gets that of v[i].
__device__ __forceinline__ float dc_sum16(float (&v)[16], int lane) {
#pragma unroll
    for (int half = 8; half > 0; half >>= 1) {
        const bool upper = lane & half;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return v[0];
}
__device__ __forceinline__ float4 dc_add4(const float4& a, const float4& b, const float4& c, const float4& d) {
    return make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y), (a.z + b.z) + (c.z + d.z), (a.w + b.w) + (c.w + d.w));
}

__device__ __forceinline__ void dc_bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(tc_smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc_smem_u32(bar)) : "memory");
}

// Chunk number `at` of the requests that are taken (in their order), by a warp; false: there is none.
__device__ __forceinline__ bool find_chunk(const int* q_start, const int* list, int requests, int at, int& row0, int& count) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int base = 0; base < requests; base += 32) {
        const bool have = base + lane < requests;
        const int r = have && list ? list[base + lane] : base + lane;
        const int first = have ? q_start[r] : 0, last = have ? q_start[r + 1] : 0;
        const int own = (max(last - first, 0) + DC_TOKENS - 1) / DC_TOKENS;
        int upto = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += u;
        }
        const unsigned reach = __ballot_sync(0xffffffffu, before + upto > at);
        if (reach) {
            const int src = __ffs(reach) - 1;
            const int index = at - before - (__shfl_sync(0xffffffffu, upto, src) - __shfl_sync(0xffffffffu, own, src));
            row0 = __shfl_sync(0xffffffffu, first, src) + index * DC_TOKENS;
            count = min(DC_TOKENS, __shfl_sync(0xffffffffu, last, src) - row0);
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// ---- 1 -----------------------------------------------------------------------------------------------------------------
// A thread owns a channel (its 16 tokens of decays, keys, queries) or a value column, but for the unit vectors (a warp per row) and
// the sums A, B: 16 lanes take columns j and 14 - j one after the other, which are 16 pairs of tokens whichever j, with the key
// of column j decaying in their registers as the rows go down. The record is put together in shared memory, in two parts that
// take turns there.
template <int D>
__global__ void __launch_bounds__(DC_PREP_THREADS, 4) delta_chunks_kernel(const DeltaChunkArgs a) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    constexpr int LD = D + 4;
    float* ks = reinterpret_cast<float*>(dc_raw);              // [16][LD]
    float* qs = ks + DC_TOKENS * LD;
    float* gs = qs + DC_TOKENS * LD;                           // decays
    unsigned char* rec = reinterpret_cast<unsigned char*>(gs + DC_TOKENS * LD);
    __shared__ __align__(16) float As[DC_TOKENS][DC_TOKENS], Ts[DC_TOKENS][DC_TOKENS];
    __shared__ float Bs[DC_TOKENS][DC_TOKENS + 1], beta[DC_TOKENS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y, kh = h / (a.H / a.G), dv = a.dv;
    pdl_wait();
    pdl_trigger();
    int row0, cnt;
    if (!find_chunk(a.q_start, a.list, a.requests, blockIdx.x, row0, cnt)) return;
    unsigned char* rec_q = rec, *rec_k = rec + D * 96, *rec_b = rec + 2 * D * 96;          // first Q, K, B and G,
    float* rec_g = reinterpret_cast<float*>(rec_b + 1536);
    unsigned char* rec_w = rec, *rec_y = rec + D * 96;                                      // then W and Y in their place
    unsigned char* to = a.scratch + ((size_t)blockIdx.x * a.H + h) * dc_record(D, dv);
    auto copy = [&](int at, int bytes, const void* from) {
        for (int i = tid; i < bytes / 16; i += DC_PREP_THREADS) reinterpret_cast<uint4*>(to + at)[i] = reinterpret_cast<const uint4*>(from)[i];
    };

    // every load first: a thread's decays and values (of its first channel and column), then the rows of k and q
    const int ch = tid % D, col = tid >= D ? tid - D : tid + DC_PREP_THREADS - D;
    float raw[DC_TOKENS], value[DC_TOKENS];
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) raw[t] = t < cnt ? a.decay[(size_t)(row0 + t) * a.decay_t + (size_t)h * D + ch] : 0.f;
#pragma unroll
    for (int t = 0; t < DC_TOKENS; ++t) value[t] = col < dv && t < cnt ? a.v[(size_t)(row0 + t) * a.v_t + (size_t)h * dv + col] : 0.f;
    constexpr int ROWS = DC_PREP_THREADS / D;                  // rows the block's threads read at once
#pragma unroll
    for (int i = 0; i < DC_TOKENS / ROWS; ++i) {
        const int t = i * ROWS + tid / D;
        ks[t * LD + ch] = t < cnt ? a.k[(size_t)(row0 + t) * a.k_t + (size_t)kh * D + ch] : 0.f;
        qs[t * LD + ch] = t < cnt ? a.q[(size_t)(row0 + t) * a.q_t + (size_t)kh * D + ch] : 0.f;
    }
    if (tid < D) {
        const float rate = -expf(a.a_log[h]), bias = a.dt_bias[(size_t)h * D + ch];
#pragma unroll
        for (int t = 0; t < DC_TOKENS; ++t) gs[t * LD + ch] = t < cnt ? expf(rate * dc_softplus(raw[t] + bias)) : 1.f;
    }
    if (tid < DC_TOKENS) beta[tid] = tid < cnt ? 1.f / (1.f + expf(-a.beta[(size_t)(row0 + tid) * a.beta_t + h])) : 0.f;
    As[tid / 16][tid % 16] = 0.f;
    As[8 + tid / 16][tid % 16] = 0.f;
    __syncthreads();
    {   // unit vectors, and B's diagonal
        const float q_scale = 1.f / sqrtf((float)D);
#pragma unroll
        for (int i = 0; i < DC_TOKENS / 4; ++i) {
            const int t = warp * (DC_TOKENS / 4) + i;
            float kk = 0.f, qq = 0.f, kq = 0.f;
#pragma unroll
            for (int c = 0; c < D; c += 32) {
                const float kv = ks[t * LD + c + lane], qv = qs[t * LD + c + lane];
                kk = fmaf(kv, kv, kk);
                qq = fmaf(qv, qv, qq);
                kq = fmaf(kv, qv, kq);
            }
            kk = warp_sum(kk);
            qq = warp_sum(qq);
            kq = warp_sum(kq);
            const float kf = 1.f / sqrtf(kk + 1e-6f), qf = q_scale / sqrtf(qq + 1e-6f);
#pragma unroll
            for (int c = 0; c < D; c += 32) {
                ks[t * LD + c + lane] *= kf;
                qs[t * LD + c + lane] *= qf;
            }
            if (lane < DC_TOKENS) Bs[t][lane] = lane == t ? kq * kf * qf : 0.f;
        }
    }
    __syncthreads();
    {   // A and B below their diagonals
        constexpr int F4 = D / 64;                             // 16-byte pieces of a row a lane takes
        const int m = tid >> 4, at = (tid & 15) * 4, turn = DC_TOKENS - 1 - m;
        float sa[DC_TOKENS], sb[DC_TOKENS];
        float4 p[F4];
        auto row = [&](const float* from, int t, int i) { return *reinterpret_cast<const float4*>(from + t * LD + i * 64 + at); };
#pragma unroll
        for (int i = 0; i < F4; ++i) p[i] = row(ks, m, i);
#pragma unroll
        for (int s = 0; s < DC_TOKENS; ++s) {                  // column m down to the last row, then column 14 - m
            const int t = s < turn ? m + 1 + s : s;
            if (s >= DC_TOKENS / 2 && s == turn) {
#pragma unroll
                for (int i = 0; i < F4; ++i) p[i] = row(ks, turn - 1, i);
            }
            sa[s] = sb[s] = 0.f;
#pragma unroll
            for (int i = 0; i < F4; ++i) {
                const float4 g = row(gs, t, i);
                p[i] = make_float4(p[i].x * g.x, p[i].y * g.y, p[i].z * g.z, p[i].w * g.w);
                sa[s] = dc_dot(row(ks, t, i), p[i], sa[s]);
                sb[s] = dc_dot(row(qs, t, i), p[i], sb[s]);
            }
        }
        const float va = dc_sum16(sa, lane), vb = dc_sum16(sb, lane);
        const int s = tid & 15, t = s < turn ? m + 1 + s : s, j = s < turn ? m : turn - 1;
        if (m < 7 || s < turn) {                               // (column 7 is its own partner)
            As[t][j] = va;
            Bs[t][j] = vb;
        }
    }
    __syncthreads();
    if (tid < 32) {
        if (lane < DC_TOKENS) {                                // column `lane` of T by forward substitution
            float x[DC_TOKENS];
#pragma unroll
            for (int t = 0; t < DC_TOKENS; ++t) {
                float s = t == lane ? 1.f : 0.f, s2 = 0.f;
#pragma unroll
                for (int i = 0; i < t; ++i) {
                    if (i & 1) s2 = fmaf(-As[t][i], x[i], s2);
                    else s = fmaf(-As[t][i], x[i], s);
                }
                x[t] = beta[t] * (s + s2);
                Ts[t][lane] = x[t];
            }
        }
    } else {                                                   // meanwhile the others: B, and Q, K, G, which need neither A nor T
        if (warp >= 2) {                                       // j along k, t along n (above the diagonal B is zero)
            const int n = warp - 2, t = n * 8 + (lane >> 2), j = (lane & 3) * 2;
            unsigned b0[3], b1[3];
            dc_split(Bs[t][j], Bs[t][j + 1], b0[0], b0[1], b0[2]);
            dc_split(Bs[t][j + 8], Bs[t][j + 9], b1[0], b1[1], b1[2]);
            dc_put(rec_b + n * DC_FRAGMENT, lane, b0, b1);
        }
        for (int c = tid - 32; c < D; c += DC_PREP_THREADS - 32) {
            float g[DC_TOKENS], kb[DC_TOKENS], upto = 1.f, after = 1.f;
#pragma unroll
            for (int t = 0; t < DC_TOKENS; ++t) g[t] = gs[t * LD + c];
#pragma unroll
            for (int t = DC_TOKENS - 1; t >= 0; --t) {
                kb[t] = ks[t * LD + c] * after;
                after *= g[t];
            }
#pragma unroll
            for (int t = 0; t < DC_TOKENS; ++t) {
                upto *= g[t];
                // B operand with channels along k and tokens along n
                dc_put(rec_q + ((c >> 4) * 2 + (t >> 3)) * DC_FRAGMENT, (t & 7) * 4 + ((c & 7) >> 1), (c >> 3) & 1, c & 1, qs[t * LD + c] * upto);
            }
            rec_g[c] = upto;
#pragma unroll
            for (int p = 0; p < 4; ++p) {                      // B operand with tokens along k and channels along n
                unsigned b0[3], b1[3];
                dc_split(kb[2 * p], kb[2 * p + 1], b0[0], b0[1], b0[2]);
                dc_split(kb[8 + 2 * p], kb[9 + 2 * p], b1[0], b1[1], b1[2]);
                dc_put(rec_k + (c >> 3) * DC_FRAGMENT, (c & 7) * 4 + p, b0, b1);
            }
        }
    }
    __syncthreads();
    copy(D * 96, 2 * D * 96 + 1536, rec_q);
    copy(3 * D * 96 + 1536 + dv * 64, D * 4, rec_g);
    __syncthreads();
    for (int i = tid; i < D + dv; i += DC_PREP_THREADS) {      // W, Y: rows of T times a channel's keys or a column's values
        const bool key = i < D;
        const int c = key ? i : i - D;
        float x[DC_TOKENS];
        if (key) {
            float upto = 1.f;
#pragma unroll
            for (int t = 0; t < DC_TOKENS; ++t) {
                upto *= gs[t * LD + c];
                x[t] = ks[t * LD + c] * upto;
            }
        } else {
#pragma unroll
            for (int t = 0; t < DC_TOKENS; ++t) {
                if (c == col) x[t] = value[t];
                else x[t] = t < cnt ? a.v[(size_t)(row0 + t) * a.v_t + (size_t)h * dv + c] : 0.f;
            }
        }
#pragma unroll
        for (int t = 0; t < DC_TOKENS; t += 2) {
            float y[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float s0 = 0.f, s1 = 0.f;
#pragma unroll
                for (int j = 0; j <= t + u; ++j) {
                    if (j & 1) s1 = fmaf(Ts[t + u][j], x[j], s1);
                    else s0 = fmaf(Ts[t + u][j], x[j], s0);
                }
                y[u] = s0 + s1;
            }
            if (key) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    dc_put(rec_w + ((c >> 4) * 2 + (t >> 3)) * DC_FRAGMENT, ((t + u) & 7) * 4 + ((c & 7) >> 1), (c >> 3) & 1, c & 1, y[u]);
            } else {                                           // accumulator with columns along m and tokens along n
                *reinterpret_cast<float2*>(rec_y + ((c >> 4) * 2 + (t >> 3)) * 512 + ((c & 7) * 4 + ((t & 7) >> 1)) * 16 + ((c >> 3) & 1) * 8) =
                    make_float2(y[0], y[1]);
            }
        }
    }
    __syncthreads();
    copy(0, D * 96, rec_w);
    copy(3 * D * 96 + 1536, dv * 64, rec_y);
}

// ---- 2 -----------------------------------------------------------------------------------------------------------------
// The state is held transposed, S^T with columns along m and channels along n: its accumulators are then, as they lie, the A
// operand of the products with W and Q, and U^T that of the products with K and B. A block has 16 value columns, a warp a quarter of
// the channels. The quarters' shares of U^T and of the outputs meet in shared memory (two buffers, one barrier a chunk), where every
// warp adds all of U^T and its part of the outputs. The records come through a ring of DC_STAGES by bulk copies; a stage is
// free once every warp is in the chunk after it.
template <int KS>
__global__ void __launch_bounds__(DC_CHAIN_THREADS) delta_chain_kernel(const DeltaChunkArgs a) {
    constexpr int D = 64 * KS, MAIN = 3 * D * 96 + 1536, STAGE = MAIN + 1024 + D * 4;
    extern __shared__ __align__(128) unsigned char dc_ring[];
    __shared__ __align__(16) float4 shares[2][4][4][32];       // [buffer][quarter][U, U, o, o][lane]
    __shared__ __align__(8) uint64_t full[DC_STAGES];
    const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int h = blockIdx.x, r = a.list ? a.list[blockIdx.z] : blockIdx.z, dv = a.dv;
    if (tid == 0) {
        for (int i = 0; i < DC_STAGES; ++i) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    pdl_wait();
    pdl_trigger();
    const int begin = a.q_start[r], tokens = a.q_start[r + 1] - begin;
    if (tokens <= 0) return;
    const int chunks = (tokens + DC_TOKENS - 1) / DC_TOKENS;
    int first = 0;
    for (int i = lane; i < blockIdx.z; i += 32) {
        const int other = a.list ? a.list[i] : i;
        first += (max(a.q_start[other + 1] - a.q_start[other], 0) + DC_TOKENS - 1) / DC_TOKENS;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
    const int bytes = dc_record(D, dv);
    const size_t stride = (size_t)a.H * bytes;
    const unsigned char* rec = a.scratch + ((size_t)first * a.H + h) * bytes;
    auto issue = [&](int s) {                                  // thread 0
        const unsigned char* at = rec + (size_t)s * stride;
        unsigned char* to = dc_ring + (s % DC_STAGES) * STAGE;
        uint64_t* bar = &full[s % DC_STAGES];
        mbar_expect_tx(bar, STAGE);
        dc_bulk_copy(to, at, MAIN, bar);
        dc_bulk_copy(to + MAIN, at + MAIN + blockIdx.y * 1024, 1024, bar);
        dc_bulk_copy(to + MAIN + 1024, at + MAIN + dv * 64, D * 4, bar);
    };
    if (tid == 0)
        for (int s = 0; s < min(chunks, DC_STAGES); ++s) issue(s);
    const int col0 = blockIdx.y * 16, c0 = part * 16 * KS;
    const int p0 = a.positions[begin];
    float* slot = a.state + (size_t)a.slots[r] * a.state_slot + (size_t)h * D * dv;
    const float* rd = slot + ((p0 + 1) & 1) * a.state_half;
    float* wr = slot + ((p0 + tokens - 1) & 1) * a.state_half;
    float S[2 * KS][4];
#pragma unroll
    for (int n = 0; n < 2 * KS; ++n) {
        const float* at = rd + (size_t)(c0 + n * 8 + 2 * t4) * dv + col0 + g;
        S[n][0] = at[0];
        S[n][1] = at[dv];
        S[n][2] = at[8];
        S[n][3] = at[dv + 8];
    }
    __syncthreads();                                           // the barriers are set up
    float* out = a.o + (size_t)begin * a.o_t + (size_t)h * dv + col0 + g;
    for (int s = 0; s < chunks; ++s) {
        const unsigned char* st = dc_ring + (s % DC_STAGES) * STAGE;
        auto fragment = [&](int i) { return dc_fragment(st + i * DC_FRAGMENT, lane); };
        mbar_wait(&full[s % DC_STAGES], (uint32_t)(s / DC_STAGES) & 1u, a.error_flag);
        float uo[4][4] = {}, rest[4][4] = {};                  // U of tokens 0 .. 7, of 8 .. 15, o likewise
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            unsigned sp[3][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) dc_split(S[2 * k + (i >> 1)][(i & 1) * 2], S[2 * k + (i >> 1)][(i & 1) * 2 + 1], sp[0][i], sp[1][i], sp[2][i]);
            const int at = (part * KS + k) * 2;
            const DcFragment wq[4] = {fragment(at), fragment(at + 1), fragment(D / 8 + at), fragment(D / 8 + at + 1)};
            dc_products(uo, rest, sp, wq);
        }
        float4 (*meet)[4][32] = shares[s & 1];
#pragma unroll
        for (int n = 0; n < 4; ++n)
            meet[part][n][lane] = make_float4(uo[n][0] + rest[n][0], uo[n][1] + rest[n][1], uo[n][2] + rest[n][2], uo[n][3] + rest[n][3]);
        __syncthreads();
        if (tid == 0 && s > 0 && s - 1 + DC_STAGES < chunks) issue(s - 1 + DC_STAGES);
        float u[2][4], none = 0.f;                             // U^T; `none`: 0, or a NaN if an entry is no finite number
        unsigned up[3][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float4 sum = dc_add4(meet[0][n][lane], meet[1][n][lane], meet[2][n][lane], meet[3][n][lane]);
            const float4 y = *reinterpret_cast<const float4*>(st + MAIN + (n * 32 + lane) * 16);
            u[n][0] = y.x - sum.x; u[n][1] = y.y - sum.y; u[n][2] = y.z - sum.z; u[n][3] = y.w - sum.w;
            dc_split(u[n][0], u[n][1], up[0][2 * n], up[1][2 * n], up[2][2 * n]);
            dc_split(u[n][2], u[n][3], up[0][2 * n + 1], up[1][2 * n + 1], up[2][2 * n + 1]);
#pragma unroll
            for (int i = 0; i < 4; ++i) none = fmaf(u[n][i], 0.f, none);
        }
        const float2* decay = reinterpret_cast<const float2*>(st + MAIN + 1024) + (c0 >> 1) + t4;
        // a quarter stores the outputs of a half of the tokens and of 8 of the columns
        const int half = part & 1, upper = part >> 1;
        DcFragment kb[2 * KS + 1];                             // K of the quarter's channels, and B
#pragma unroll
        for (int n = 0; n < 2 * KS; ++n) kb[n] = fragment(2 * D / 8 + part * 2 * KS + n);
        kb[2 * KS] = fragment(3 * D / 8 + half);
        float big[2 * KS + 1][4] = {}, small[2 * KS + 1][4] = {};
        dc_products(big, small, up, kb);
#pragma unroll
        for (int n = 0; n < 2 * KS; ++n) {
            const float2 d = decay[n * 4];
#pragma unroll
            for (int i = 0; i < 4; ++i) S[n][i] = fmaf(S[n][i], i & 1 ? d.y : d.x, big[n][i] + small[n][i]);
        }
        const float4 sum = dc_add4(meet[0][2 + half][lane], meet[1][2 + half][lane], meet[2][2 + half][lane], meet[3][2 + half][lane]);
        float y[4] = {sum.x, sum.y, sum.z, sum.w};
        if (__any_sync(0xffffffffu, none != none)) {           // a zero of B above its diagonal times what is no number would be none
            float v[2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[n][i] = fabsf(u[n][i]) < INFINITY ? u[n][i] : 0.f;
                dc_split(v[n][0], v[n][1], up[0][2 * n], up[1][2 * n], up[2][2 * n]);
                dc_split(v[n][2], v[n][3], up[0][2 * n + 1], up[1][2 * n + 1], up[2][2 * n + 1]);
            }
            float b[1][4] = {}, r[1][4] = {};
            const DcFragment only[1] = {kb[2 * KS]};
            dc_products(b, r, up, only);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                y[i] += b[0][i] + r[0][i];
#pragma unroll
                for (int j = 0; j < DC_TOKENS; ++j) {          // and such entries of tokens up to the output's own, in column g + 8 (i / 2)
                    const float uj = __shfl_sync(0xffffffffu, u[j >> 3][(i & 2) + (j & 1)], g * 4 + ((j & 7) >> 1));
                    if (j <= half * 8 + 2 * t4 + (i & 1) && !(fabsf(uj) < INFINITY)) y[i] += uj;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] += big[2 * KS][i] + small[2 * KS][i];
        }
        const int t = s * DC_TOKENS + half * 8 + 2 * t4;
        float* to = out + (size_t)t * a.o_t + upper * 8;
        if (t < tokens) to[0] = upper ? y[2] : y[0];
        if (t + 1 < tokens) to[a.o_t] = upper ? y[3] : y[1];
    }
#pragma unroll
    for (int n = 0; n < 2 * KS; ++n) {
        float* at = wr + (size_t)(c0 + n * 8 + 2 * t4) * dv + col0 + g;
        at[0] = S[n][0];
        at[dv] = S[n][1];
        at[8] = S[n][2];
        at[dv + 8] = S[n][3];
    }
}

template <int KS> void launch_chunks(const DeltaChunkArgs& a, int chunks, cudaStream_t stream) {
    constexpr int D = 64 * KS;
    const int part1 = 2 * D * 96 + 1536 + D * 4, part2 = D * 96 + a.dv * 64;
    const size_t smem = (size_t)3 * DC_TOKENS * (D + 4) * sizeof(float) + (part1 > part2 ? part1 : part2);
    LLMP_ALLOW_SMEM(delta_chunks_kernel<D>, smem);
    llmp_launch_dependent(delta_chunks_kernel<D>, dim3(chunks, a.H), dim3(DC_PREP_THREADS), smem, stream, a);
    const size_t ring = (size_t)DC_STAGES * (3 * D * 96 + 1536 + 1024 + D * 4);
    LLMP_ALLOW_SMEM(delta_chain_kernel<KS>, ring);
    llmp_launch_dependent(delta_chain_kernel<KS>, dim3(a.H, a.dv / 16, a.requests), dim3(DC_CHAIN_THREADS), ring, stream, a);
}

}  // namespace

// delta_rule.cu
LLMP_API int llmp_delta_prep(float* q, long q_t, float* k, long k_t, float* decay, long decay_t, float* beta, long beta_t, const float* a_log,
                             const float* dt_bias, const int* token_request, const int* q_start, int least, int max_tokens, int tokens, int H, int G, int d,
                             cudaStream_t stream);
LLMP_API int llmp_delta_scan(const float* q, long q_t, const float* k, long k_t, const float* v, long v_t, const float* decay, long decay_t,
                             const float* beta, long beta_t, float* state, long state_slot, long state_half, const int* q_start, const int* slots,
                             const int* positions, float* o, long o_t, int least, int max_tokens, int R, int H, int G, int d, int dv, cudaStream_t stream);

// Bytes of scratch for `rows` tokens of R requests; 0: these sizes are not served.
LLMP_API long llmp_delta_chunks_scratch(int rows, int R, int H, int d, int dv) {
    if (rows <= 0 || R <= 0 || H <= 0 || (d != 64 && d != 128) || dv < 16 || dv % 16 || dv > 512) return 0;
    return ((long)(rows - 1) / DC_TOKENS + R) * H * dc_record(d, dv);
}

// q, k, v: the convolved rows; decay, beta: pre-activations (delta_prep and delta_scan in one). list: `count` of the R requests, in
// ascending order, which have `rows` of the step's tokens together; the others, which have up to max_tokens each, go token by token
// (their rows are prepared in place), those of fewer than `least` are left alone. null: all requests in chunks.
LLMP_API int llmp_delta_chunks(float* q, long q_t, float* k, long k_t, const float* v, long v_t, float* decay, long decay_t,
                               float* beta, long beta_t, const float* a_log, const float* dt_bias, float* state, long state_slot,
                               long state_half, const int* q_start, const int* slots, const int* positions, float* o, long o_t, void* scratch,
                               long scratch_bytes, const int* list, int count, int rows, const int* token_request, int least, int max_tokens, int tokens,
                               int R, int H, int G, int d, int dv, int* error_flag, cudaStream_t stream) {
    if (R <= 0 || tokens <= 0) return 0;
    LLMP_REQUIRE(rows > 0 && rows <= tokens && count > 0 && count <= R && (list ? token_request != nullptr : count == R && rows == tokens),
                 "delta_chunks: %d of %d requests, %d of %d tokens", count, R, rows, tokens);
    LLMP_REQUIRE(H > 0 && G > 0 && H % G == 0 && H <= 65535 && R <= 65535, "delta_chunks: bad sizes heads=%d qk_heads=%d requests=%d", H, G, R);
    LLMP_REQUIRE(error_flag != nullptr, "delta_chunks: an error flag in device memory is required");
    const long need = llmp_delta_chunks_scratch(rows, count, H, d, dv);
    LLMP_REQUIRE(need > 0, "delta_chunks: heads of %d x %d are not served", d, dv);
    LLMP_REQUIRE(scratch != nullptr && scratch_bytes >= need && (size_t)scratch % 16 == 0, "delta_chunks: %ld bytes of scratch are needed", need);
    DeltaChunkArgs a;
    a.q = q; a.q_t = q_t; a.k = k; a.k_t = k_t; a.v = v; a.v_t = v_t; a.decay = decay; a.decay_t = decay_t; a.beta = beta; a.beta_t = beta_t;
    a.a_log = a_log; a.dt_bias = dt_bias; a.state = state; a.state_slot = state_slot; a.state_half = state_half; a.q_start = q_start;
    a.slots = slots; a.positions = positions; a.o = o; a.o_t = o_t; a.scratch = (unsigned char*)scratch; a.list = list; a.requests = count;
    a.H = H; a.G = G; a.dv = dv; a.error_flag = error_flag;
    const int chunks = (rows - 1) / DC_TOKENS + count;
    if (d == 64) launch_chunks<1>(a, chunks, stream);
    else launch_chunks<2>(a, chunks, stream);
    if (list && least <= max_tokens) {
        const int failed = llmp_delta_prep(q, q_t, k, k_t, decay, decay_t, beta, beta_t, a_log, dt_bias, token_request, q_start, least, max_tokens, tokens,
                                           H, G, d, stream);
        if (failed) return failed;
        return llmp_delta_scan(q, q_t, k, k_t, v, v_t, decay, decay_t, beta, beta_t, state, state_slot, state_half, q_start, slots, positions, o, o_t,
                               least, max_tokens, R, H, G, d, dv, stream);
    }
    return llmp_check_launch("delta_chunks");
}
