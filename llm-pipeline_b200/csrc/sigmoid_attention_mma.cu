// Sigmoid attention with mixed heads on the tensor cores (mma.sync m16n8k16, bfloat16 operands, float32 accumulate),
// with the contract of llmp_sigmoid_attention for bfloat16 pages and up to SM_MAX_HEADS query heads.
//
// A block takes a tile of up to 16 consecutive new tokens of one request and one range of keys, with a warp per
// query head. Keys are walked in tiles of 32 aligned to key 0. For a key tile
//   1. warp g multiplies its head's 16 queries with the 32 keys of its key/value head, caps the scores, takes the
//      sigmoid (float32) and leaves the 16 x 32 weights in shared memory, the pairs in the order of its registers;
//   2. the weights of all heads are mixed by the matrix of the heads as a product of its own: 16 heads out, 16 heads in, a column
//      for each of the 512 (token, key) pairs, dealt out over the warps. Both factors are split into three bfloat16 pieces, which
//      hold all 24 bits, and the six larger products of pieces summed in float32: rows of the matrix may cancel;
//   3. they are rounded to bfloat16, and warp h multiplies those of its head with the 32 values of its key/value head.
// Nothing is normalised over keys, so the output registers simply add up over key tiles and key ranges: with more
// than one range the blocks leave float32 partial sums that a second kernel adds in the order of the ranges.
// The keys of the next tile are copied (cp.async) while the weights are mixed and multiplied with the values, the
// values of the next tile while the next scores are made.
// With every warp adding up all heads' float32 weights on the CUDA cores, a key tile moved 512 KB through shared memory for the
// mix alone, 4,096 clocks of an SM; as a product it moves 100 KB. 2,048 tokens of 16 heads of 128: 285 us before, 197 with the
// product, 168 with tanh as a series where the scores are far below the cap, exponentials and reciprocals without their range
// checks, masks only where a row's end is near, and a tile's places found a tile ahead (three pieces instead of two: a layer 230
// -> 240). What is left is the latency of four phases between barriers at four warps a scheduler (issue slots 44 %, tensor
// pipe 30 %). Shorter key ranges (512, 256 keys) lose to their partial sums: 205, 222 us against 197.
#include "common.cuh"

namespace {

constexpr int SM_MAX_HEADS = 16;
constexpr int SM_ROWS = 16;
constexpr int SM_KEYS = 32;

struct SigMmaArgs {
    const bf16* q; long q_t;
    const bf16* pages;
    const int* tables; int width;
    const int* q_start; const int* ctx_len;
    const int* tile_req; const int* tile_tok0; int num_tiles;
    const float* talk; const float* pb;
    bf16* out; long out_t;
    float* partial;
    int H, G, page_size, segments, segment_keys;
    float scale, cap;
    bool late_keys;             // the mixed weights lie where the keys do
};

__device__ __forceinline__ void sm_cp_async_16(void* smem_dst, const void* gmem_src, bool valid) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem_src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void sm_ldmatrix_x4(unsigned (&r)[4], const void* smem_ptr) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem_ptr);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__device__ __forceinline__ void sm_ldmatrix_x4_trans(unsigned (&r)[4], const void* smem_ptr) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem_ptr);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__device__ __forceinline__ void sm_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned sm_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

// Two floats as three pairs of bfloat16 that add up to them.
__device__ __forceinline__ void sm_split(float u, float v, unsigned& hi, unsigned& mid, unsigned& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(u, v);
    const float ru = u - __low2float(h), rv = v - __high2float(h);
    const __nv_bfloat162 m = __floats2bfloat162_rn(ru, rv);
    const __nv_bfloat162 l = __floats2bfloat162_rn(ru - __low2float(m), rv - __high2float(m));
    hi = *reinterpret_cast<const unsigned*>(&h);
    mid = *reinterpret_cast<const unsigned*>(&m);
    lo = *reinterpret_cast<const unsigned*>(&l);
}

__device__ __forceinline__ float sm_ex2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float sm_rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
constexpr float SM_LOG2_E = 1.4426950408889634f;
// tanh(x). SMALL: |x| <= SM_SMALL, where five terms of its series leave 2.4e-7 of the result and no work for the special-function
// unit; else 1 - 2 / (1 + e^(2x)) with an exponential whose relative error is about 2^-21.
constexpr float SM_SMALL = 0.35f;
template <bool SMALL> __device__ __forceinline__ float sm_tanh(float x) {
    if (!SMALL) return fmaf(-2.f, sm_rcp(1.f + sm_ex2(2.f * SM_LOG2_E * x)), 1.f);
    const float y = x * x;
    return x * fmaf(y, fmaf(y, fmaf(y, fmaf(y, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f), 1.f);
}
// The sigmoid of a number given times -log2(e); the exponential's and the reciprocal's errors leave the weight's near 1e-7.
__device__ __forceinline__ float sm_sigmoid(float minus_log2) { return sm_rcp(1.f + sm_ex2(minus_log2)); }

constexpr int SM_PAIRS = SM_ROWS * SM_KEYS + 4;        // a head's weights in shared memory: neighbouring heads' lie 4 banks apart
constexpr int SM_PS = SM_KEYS + 8;                     // of a token's mixed weights
constexpr int SM_PH = SM_ROWS * SM_PS + 8;             // of a head's: eight heads' rows meet no bank twice

// D16: dim / 16, DV16: vdim / 16. One warp per query head.
template <int D16, int DV16>
__global__ void __launch_bounds__(SM_MAX_HEADS * 32, 1) sigmoid_attention_mma_kernel(const SigMmaArgs a) {
    extern __shared__ __align__(16) unsigned char sm_smem[];
    constexpr int D = D16 * 16, DV = DV16 * 16;
    constexpr int KS = D + 8, VS = DV + 8;                          // padded rows: conflict-free ldmatrix
    const int H = a.H, G = a.G, hpg = H / G, rs = D + DV;
    bf16* Qs = reinterpret_cast<bf16*>(sm_smem);                    // [H][16][KS]
    bf16* Ks = Qs + (size_t)H * SM_ROWS * KS;                       // [G][32][KS]
    bf16* Vs = Ks + (size_t)G * SM_KEYS * KS;                       // [G][32][VS]
    const int wrows = min(SM_MAX_HEADS, H + 1);
    float* Ws = reinterpret_cast<float*>(Vs + (size_t)G * SM_KEYS * VS);    // [wrows][SM_PAIRS]: the weights; row H, if any, is zero
    bf16* Ps = a.late_keys ? Ks : reinterpret_cast<bf16*>(Ws + wrows * SM_PAIRS);   // [H][16][SM_PS] with SM_PH entries a head: the mixed weights
    __shared__ long long key_off[2][SM_KEYS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x;
    const int gr = lane >> 2, t = lane & 3;
    const int tile = a.num_tiles - 1 - (int)blockIdx.x;             // the tiles that see most keys start first
    const int seg = blockIdx.y;
    pdl_wait();                                    // what the kernels before wrote is complete
    pdl_trigger();
    const int r = a.tile_req[tile], tok0 = a.tile_tok0[tile];
    const int q_begin = a.q_start[r];
    const int q_len = a.q_start[r + 1] - q_begin;
    const int pos0 = a.ctx_len[r] - q_len;
    int ntok = q_len - tok0;
    if (ntok > SM_ROWS) ntok = SM_ROWS;
    const int first = q_begin + tok0;                               // the tile's first row among the step's tokens
    int lo = 0, hi = pos0 + tok0 + ntok - 1;                        // keys of this block (inclusive)
    if (a.segments > 1) {
        lo = seg * a.segment_keys;
        hi = min(hi, lo + a.segment_keys - 1);
        if (lo > hi) return;                                        // nothing of this range is visible: its sums are never read
    }
    const int* table = a.tables + (size_t)r * a.width;

    constexpr int QV = D / 8, VV = DV / 8;
    for (int e = tid; e < H * SM_ROWS * QV; e += nthreads) {
        const int c = (e % QV) * 8, row = (e / QV) % SM_ROWS, h = e / (QV * SM_ROWS);
        const bool ok = row < ntok;
        sm_cp_async_16(Qs + ((size_t)h * SM_ROWS + row) * KS + c, ok ? a.q + (size_t)(first + row) * a.q_t + (size_t)h * D + c : a.q, ok);
    }
    for (int i = tid; i < (wrows - H) * SM_PAIRS; i += nthreads) Ws[H * SM_PAIRS + i] = 0.f;
    unsigned mix[3][4];                                             // the mixing matrix as an A operand: heads out along m, heads in along k
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int ho = gr + 8 * (i & 1), hi = 2 * t + 8 * (i >> 1);
        sm_split(ho < H && hi < H ? a.talk[ho * H + hi] : 0.f, ho < H && hi + 1 < H ? a.talk[ho * H + hi + 1] : 0.f, mix[0][i], mix[1][i], mix[2][i]);
    }
    // Where the keys of a tile lie among the pages (-1: nowhere), found a tile ahead by the first warp; a barrier lies between.
    auto find_keys = [&](int j0) {
        if (tid < SM_KEYS) {
            const int j = j0 + tid;
            long long off = -1;
            if (j <= hi) {
                const int page = table[j / a.page_size];
                if (page >= 0) off = (long long)(((size_t)page * G) * a.page_size + (j % a.page_size)) * rs;
            }
            key_off[(j0 / SM_KEYS) & 1][tid] = off;
        }
    };
    // A thread copies piece `tid % pieces` of every (threads / pieces)-th row of the tile's [key/value head][key].
    const size_t head_step = (size_t)a.page_size * rs;
    auto copy_rows = [&](int j0, bf16* dst, int stride, int pieces, int from) {
        if (j0 <= hi) {
            const int step = nthreads / pieces, c = tid % pieces * 8, row0 = tid / pieces;
            const long long* offs = key_off[(j0 / SM_KEYS) & 1];
            if (row0 < step)
                for (int row = row0; row < G * SM_KEYS; row += step) {
                    const long long off = offs[row % SM_KEYS];
                    sm_cp_async_16(dst + (size_t)row * stride + c, off >= 0 ? a.pages + off + (row / SM_KEYS) * head_step + from + c : a.pages, off >= 0);
                }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto issue_keys = [&](int j0) { copy_rows(j0, Ks, KS, QV, 0); };
    auto issue_values = [&](int j0) { copy_rows(j0, Vs, VS, VV, D); };

    const int h = warp;                                             // this warp's head, in all three steps
    const int kvh = h / hpg;
    int row_pos[2];
    row_pos[0] = gr < ntok ? pos0 + tok0 + gr : -1;
    row_pos[1] = gr + 8 < ntok ? pos0 + tok0 + gr + 8 : -1;
    // a weight is sm_sigmoid(x slope + shift), with x the score or, under a cap, tanh(score to_cap)
    const float to_cap = a.cap > 0.f ? a.scale / a.cap : 0.f, slope = -SM_LOG2_E * (a.cap > 0.f ? a.cap : a.scale), shift = -SM_LOG2_E * a.pb[h];
    float o[2 * DV16][4];
#pragma unroll
    for (int i = 0; i < 2 * DV16; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

    const int tile_lo = (lo / SM_KEYS) * SM_KEYS;                   // lo is a multiple of the key tile anyway
    find_keys(tile_lo);
    __syncthreads();
    issue_keys(tile_lo);                                            // group: the queries and the first keys
    issue_values(tile_lo);
    const bf16* Qw = Qs + ((size_t)h * SM_ROWS + (lane & 15)) * KS + (lane >> 4) * 8;
    const bf16* Kw = Ks + (size_t)kvh * SM_KEYS * KS;
    const bf16* Vw = Vs + (size_t)kvh * SM_KEYS * VS;
    for (int j0 = tile_lo; j0 <= hi; j0 += SM_KEYS) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");     // this tile's keys are here
        __syncthreads();
        find_keys(j0 + SM_KEYS);                                    // (nobody reads the other half any more)
        float s[4][4];
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) s[nb][0] = s[nb][1] = s[nb][2] = s[nb][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < D16; ++ks) {
            unsigned qa[4];
            sm_ldmatrix_x4(qa, Qw + ks * 16);
#pragma unroll
            for (int nb = 0; nb < 4; nb += 2) {
                unsigned kf[4];
                sm_ldmatrix_x4(kf, Kw + (size_t)((nb + (lane >> 4)) * 8 + (lane & 7)) * KS + ks * 16 + ((lane >> 3) & 1) * 8);
                sm_mma(s[nb], qa, kf[0], kf[1]);
                sm_mma(s[nb + 1], qa, kf[2], kf[3]);
            }
        }
        if (a.cap > 0.f) {
            float top = 0.f;                                        // a NaN is one either way
#pragma unroll
            for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[nb][c] *= to_cap;
                    top = fmaxf(top, fabsf(s[nb][c]));
                }
            if (__all_sync(0xffffffffu, top <= SM_SMALL)) {
#pragma unroll
                for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                    for (int c = 0; c < 4; ++c) s[nb][c] = sm_tanh<true>(s[nb][c]);
            } else {
#pragma unroll
                for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                    for (int c = 0; c < 4; ++c) s[nb][c] = sm_tanh<false>(s[nb][c]);
            }
        }
#pragma unroll
        for (int nb = 0; nb < 4; ++nb)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[nb][c] = sm_sigmoid(fmaf(s[nb][c], slope, shift));
        if (ntok < SM_ROWS || j0 + SM_KEYS - 1 > pos0 + tok0) {     // some row does not see all of these keys
#pragma unroll
            for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (j0 + nb * 8 + 2 * t + (c & 1) > row_pos[c >> 1]) s[nb][c] = 0.f;
        }
        // the pairs of token gr + 8 hr and keys nb 8 .. of the tile are columns (2 nb + hr) 64 + 8 gr ..: a warp writes 128 bytes
        {
            float2* w = reinterpret_cast<float2*>(Ws + h * SM_PAIRS) + lane;
#pragma unroll
            for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                for (int hr = 0; hr < 2; ++hr) w[(2 * nb + hr) * 32] = make_float2(s[nb][2 * hr], s[nb][2 * hr + 1]);
        }
        __syncthreads();                                            // all weights are in place, the keys are free
        if (!a.late_keys) issue_keys(j0 + SM_KEYS);
        // 32 times 16 columns over the warps: the mixed weights of all heads for two tokens and 8 keys each
        for (int pair = warp; pair < 32; pair += H) {
            unsigned b[2][3][2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {                           // this lane's heads in: 2 t, 2 t + 1 and eight further
                const float* w0 = Ws + min(2 * t + 8 * k, wrows - 1) * SM_PAIRS + pair * 16 + gr;      // heads past H: the zero row
                const float* w1 = Ws + min(2 * t + 8 * k + 1, wrows - 1) * SM_PAIRS + pair * 16 + gr;
#pragma unroll
                for (int n = 0; n < 2; ++n) sm_split(w0[8 * n], w1[8 * n], b[n][0][k], b[n][1][k], b[n][2][k]);
            }
            float m[2][4] = {};
            constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};      // the smaller products first
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int n = 0; n < 2; ++n) sm_mma(m[n], mix[PA[i]], b[n][PB[i]][0], b[n][PB[i]][1]);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int q = pair * 2 + n, token = (q & 7) + 8 * ((q >> 3) & 1), key = (q >> 4) * 8 + 2 * t;
                if (gr < H) *reinterpret_cast<unsigned*>(Ps + gr * SM_PH + token * SM_PS + key) = sm_pack(m[n][0], m[n][1]);
                if (gr + 8 < H) *reinterpret_cast<unsigned*>(Ps + (gr + 8) * SM_PH + token * SM_PS + key) = sm_pack(m[n][2], m[n][3]);
            }
        }
        if (!a.late_keys) asm volatile("cp.async.wait_group 1;\n" ::: "memory");     // this tile's values are here
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            unsigned pa[4];
            sm_ldmatrix_x4(pa, Ps + h * SM_PH + (lane & 15) * SM_PS + kk * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int nb2 = 0; nb2 < DV16; ++nb2) {
                unsigned v[4];
                sm_ldmatrix_x4_trans(v, Vw + (size_t)(kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * VS + nb2 * 16 + (lane >> 4) * 8);
                sm_mma(o[nb2 * 2], pa, v[0], v[1]);
                sm_mma(o[nb2 * 2 + 1], pa, v[2], v[3]);
            }
        }
        __syncthreads();                                            // the values and the weights are free
        if (a.late_keys) issue_keys(j0 + SM_KEYS);
        issue_values(j0 + SM_KEYS);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");

#pragma unroll
    for (int h2 = 0; h2 < 2; ++h2) {
        if (row_pos[h2] < 0) continue;
        const size_t n = (size_t)first + gr + 8 * h2;
        if (a.segments > 1) {
            float* dst = a.partial + (n * a.segments + seg) * H * DV + (size_t)h * DV + 2 * t;
#pragma unroll
            for (int nb = 0; nb < 2 * DV16; ++nb) *reinterpret_cast<float2*>(dst + nb * 8) = make_float2(o[nb][2 * h2], o[nb][2 * h2 + 1]);
        } else {
            bf16* dst = a.out + n * a.out_t + (size_t)h * DV + 2 * t;
#pragma unroll
            for (int nb = 0; nb < 2 * DV16; ++nb) *reinterpret_cast<unsigned*>(dst + nb * 8) = sm_pack(o[nb][2 * h2], o[nb][2 * h2 + 1]);
        }
    }
}

// Shared memory with the mixed weights in a place of their own or (`late_keys`) in that of the keys, whose copies then wait for the
// values' product: for sizes that would not fit otherwise.
size_t sm_smem_bytes(int H, int G, int d, int dv, bool late_keys) {
    const size_t keys = (size_t)G * SM_KEYS * (d + 8), mixed = (size_t)H * SM_PH;
    return sizeof(bf16) * ((size_t)H * SM_ROWS * (d + 8) + keys + (size_t)G * SM_KEYS * (dv + 8) + (late_keys ? 0 : mixed)) +
           sizeof(float) * (size_t)(H < SM_MAX_HEADS ? H + 1 : H) * SM_PAIRS;
}
constexpr size_t SM_MOST_BYTES = 226 * 1024;
bool sm_late_keys(int H, int G, int d, int dv) {
    return sm_smem_bytes(H, G, d, dv, false) > SM_MOST_BYTES && (size_t)G * SM_KEYS * (d + 8) >= (size_t)H * SM_PH;
}

}  // namespace

namespace {

// out[n, c] = sum over the key ranges that hold a visible key of partial[n, range, c], in their order; four columns a thread (value
// sizes are multiples of 16).
__global__ void __launch_bounds__(256) sigmoid_mma_ranges_kernel(const float* __restrict__ partial, const int* __restrict__ positions,
                                                                 bf16* __restrict__ out, long out_t, int W, int segments, int segment_keys) {
    pdl_wait();                                    // what the kernels before wrote is complete
    pdl_trigger();
    const int n = blockIdx.x;
    const int used = min(segments, positions[n] / segment_keys + 1);
    for (int c = threadIdx.x * 4; c < W; c += blockDim.x * 4) {
        const float* at = partial + (size_t)n * segments * W + c;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < used; ++k) {
            const float4 v = *reinterpret_cast<const float4*>(at + (size_t)k * W);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        unsigned* o = reinterpret_cast<unsigned*>(out + (size_t)n * out_t + c);
        o[0] = sm_pack(s.x, s.y);
        o[1] = sm_pack(s.z, s.w);
    }
}

}  // namespace

// Whether the tensor-core kernel takes these sizes (bfloat16 only).
LLMP_API int llmp_sigmoid_attention_mma_supports(int H, int G, int d, int dv) {
    if (H <= 0 || G <= 0 || H % G || H > SM_MAX_HEADS) return 0;
    auto instance = [](int x) { return x == 16 || x == 32 || x == 64 || x == 96 || x == 128; };
    if (!instance(d) || !instance(dv)) return 0;
    return sm_smem_bytes(H, G, d, dv, sm_late_keys(H, G, d, dv)) <= SM_MOST_BYTES ? 1 : 0;
}

LLMP_API int llmp_sigmoid_attention_mma(const void* q, long q_t, const void* pages, const int* tables, int width, const int* q_start,
                                        const int* ctx_len, const int* positions, const int* tile_req, const int* tile_tok0,
                                        int num_tiles, const float* talk, const float* pb, void* out, long out_t, float* partial,
                                        int segments, int segment_keys, int N, int H, int G, int d, int dv, int page_size,
                                        float scale, float cap, cudaStream_t stream) {
    if (N <= 0 || num_tiles <= 0) return 0;
    LLMP_REQUIRE(llmp_sigmoid_attention_mma_supports(H, G, d, dv), "sigmoid_attention_mma: no kernel for heads=%d kv_heads=%d dim=%d vdim=%d",
                 H, G, d, dv);
    LLMP_REQUIRE(page_size > 0 && width > 0 && q_t % 8 == 0 && out_t % 2 == 0, "sigmoid_attention_mma: page=%d width=%d, rows must be 16-byte aligned",
                 page_size, width);
    LLMP_REQUIRE(segments >= 1 && segments <= 65535 && (segments == 1 || (partial && segment_keys > 0 && segment_keys % SM_KEYS == 0)),
                 "sigmoid_attention_mma: %d key ranges of %d keys", segments, segment_keys);
    SigMmaArgs a;
    a.q = (const bf16*)q; a.q_t = q_t; a.pages = (const bf16*)pages; a.tables = tables; a.width = width; a.q_start = q_start;
    a.ctx_len = ctx_len; a.tile_req = tile_req; a.tile_tok0 = tile_tok0; a.num_tiles = num_tiles; a.talk = talk; a.pb = pb;
    a.out = (bf16*)out; a.out_t = out_t; a.partial = partial; a.H = H; a.G = G; a.page_size = page_size; a.segments = segments;
    a.segment_keys = segments > 1 ? segment_keys : 0; a.scale = scale; a.cap = cap;
    a.late_keys = sm_late_keys(H, G, d, dv);
    const size_t smem = sm_smem_bytes(H, G, d, dv, a.late_keys);
    dim3 grid(num_tiles, segments);
#define LLMP_SM_CASE(A, B)                                                                   \
    if (d == 16 * A && dv == 16 * B) {                                                       \
        LLMP_ALLOW_SMEM((sigmoid_attention_mma_kernel<A, B>), smem);                         \
        llmp_launch_dependent(sigmoid_attention_mma_kernel<A, B>, grid, dim3(H * 32), smem, stream, a); \
    } else
#define LLMP_SM_ROW(A) LLMP_SM_CASE(A, 1) LLMP_SM_CASE(A, 2) LLMP_SM_CASE(A, 4) LLMP_SM_CASE(A, 6) LLMP_SM_CASE(A, 8)
    LLMP_SM_ROW(1) LLMP_SM_ROW(2) LLMP_SM_ROW(4) LLMP_SM_ROW(6) LLMP_SM_ROW(8)
    {
        llmp_set_error("sigmoid_attention_mma: dim=%d vdim=%d has no instance", d, dv);
        return 1;
    }
#undef LLMP_SM_ROW
#undef LLMP_SM_CASE
    if (segments > 1)
        llmp_launch_dependent(sigmoid_mma_ranges_kernel, dim3(N), dim3(256), 0, stream, (const float*)partial, positions, (bf16*)out, out_t, H * dv, segments,
                              segment_keys);
    return llmp_check_launch("sigmoid_attention_mma");
}
