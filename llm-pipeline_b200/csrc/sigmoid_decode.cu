// Sigmoid attention with mixed heads for steps of single tokens (bfloat16 pages, mma.sync with float32 sums), with the contract of
// llmp_sigmoid_attention. The tiles of 16 tokens of sigmoid_attention_mma.cu hold one token there and walk 32 keys at a time through
// four barriers; here the rows of a product are the query heads of a group, and a block takes KT = 64 (or 32) keys of one
// token and a range at a time, for all heads:
//   1. scores: a warp multiplies the queries of a group with 8 of its keys at a time, caps, takes the sigmoid and leaves the
//      float32 weights in shared memory;
//   2. mix: a thread adds up all heads' weights of a key for some of the heads (float32), rounds them once to bfloat16;
//   3. values: a warp multiplies a group's mixed weights with 16 columns of its values at a time.
// All keys and values of the first tile are asked for at once; in a longer range the keys of the next tile are copied from the mix on,
// its values after the products. Nothing is normalised, so ranges are sums that a second kernel adds in a fixed order, a block per 128
// columns of a row. 8 requests of 2,000 keys, 16 heads over 4 of 128 + 128: attention and sums 28 us there, 15 here (ranges of 128
// keys, so that the blocks, of which each fills an SM, are one round; ranges of 64 keys 17, of 192 19.5). The layer chooses the ranges.
#include "common.cuh"

namespace {

constexpr int SD_THREADS = 512, SD_WARPS = 16, SD_MAX_HEADS = 16, SD_PIECES = 4;      // pieces of 16 value columns that a warp holds at most

struct SigDecodeArgs {
    const bf16* q; long q_t;
    const bf16* pages;
    const int* tables; int width;
    const int* ctx_len;
    const float* talk; const float* pb;
    bf16* out; long out_t;
    float* partial;                       // null: one range
    int H, G, D, DV, page_size, segments, segment_keys;
    float scale, cap;
};

__device__ __forceinline__ void sd_copy(void* dst, const void* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void sd_x4(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void sd_x2(unsigned& r0, unsigned& r1, const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
__device__ __forceinline__ void sd_x4_trans(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void sd_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned sd_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

// Shared memory, in this order: queries [G][16][D + 8], keys [G][KT][D + 8], values [G][KT][DV + 8], mixed weights [G][16][KT + 8] (all
// bfloat16), weights [H][KT + 8] and the mixing matrix [H][H] in float32.
__host__ __device__ constexpr size_t sd_smem(int H, int G, int D, int DV, int KT) {
    return 2 * ((size_t)G * 16 * (D + 8) + (size_t)G * KT * (D + DV + 16) + (size_t)G * 16 * (KT + 8)) + 4 * ((size_t)H * (KT + 8) + H * H);
}

__device__ __forceinline__ float sd_ex2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float sd_rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
constexpr float SD_LOG2_E = 1.4426950408889634f;
// tanh as in sigmoid_attention_mma.cu: near zero five terms of its series (2.4e-7 of the result), else by the special-function unit.
__device__ __forceinline__ float sd_tanh(float x) {
    const float y = x * x;
    const float near = x * fmaf(y, fmaf(y, fmaf(y, fmaf(y, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f), 1.f);
    const float far = fmaf(-2.f, sd_rcp(1.f + sd_ex2(2.f * SD_LOG2_E * x)), 1.f);
    return fabsf(x) <= 0.35f ? near : far;
}

// D16, DV16: dim / 16 and vdim / 16, or 0 for sizes that are known at run time only.
template <int KT, int D16, int DV16>
__global__ void __launch_bounds__(SD_THREADS, 1) sigmoid_decode_kernel(const SigDecodeArgs a) {
    extern __shared__ __align__(16) unsigned char sd_raw[];
    const int H = a.H, G = a.G, D = D16 ? 16 * D16 : a.D, DV = DV16 ? 16 * DV16 : a.DV, hpg = H / G, rs = D + DV, KS = D + 8, VS = DV + 8;
    constexpr int PS = KT + 8;
    bf16* const Qs = reinterpret_cast<bf16*>(sd_raw);
    bf16* const Ks = Qs + G * 16 * KS;
    bf16* const Vs = Ks + G * KT * KS;
    bf16* const Ps = Vs + G * KT * VS;
    float* const Ws = reinterpret_cast<float*>(Ps + G * 16 * PS);
    float* const mix = Ws + H * PS;
    __shared__ long long key_off[KT];
    __shared__ float bias[SD_MAX_HEADS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int n = blockIdx.x;
    for (int i = tid; i < H * H; i += SD_THREADS) mix[i] = a.talk[i];      // weights: nothing of the step writes them
    if (tid < H) bias[tid] = -SD_LOG2_E * a.pb[tid];
    for (int i = tid; i < G * 16 * PS / 2; i += SD_THREADS) reinterpret_cast<unsigned*>(Ps)[i] = 0u;
    pdl_wait();
    pdl_trigger();
    const int last = a.ctx_len[n] - 1;
    const int lo = blockIdx.y * a.segment_keys, hi = a.partial ? min(last, lo + a.segment_keys - 1) : last;
    if (lo > hi) return;                                         // the token does not see this range: its sums are never read
    const int* table = a.tables + (size_t)n * a.width;
    const size_t head_step = (size_t)a.page_size * rs;
    auto place = [&](int j) -> long long {
        if (j > hi) return -1;
        const int page = table[j / a.page_size];
        return page >= 0 ? (long long)(((size_t)page * G) * a.page_size + j % a.page_size) * rs : -1;
    };
    if (tid < KT) key_off[tid] = place(lo + tid);
    const int qv = D / 8, vv = DV / 8;
    for (int e = tid; e < G * 16 * qv; e += SD_THREADS) {
        const int c = e % qv * 8, row = e / qv % 16, group = e / (qv * 16);
        const bool ok = row < hpg;
        sd_copy(Qs + (group * 16 + row) * KS + c, ok ? a.q + (size_t)n * a.q_t + (size_t)(group * hpg + row) * D + c : a.q, ok);
    }
    // a thread copies the same 16-byte piece of every (threads / pieces)-th row of the tile's [group][key]
    auto copy_rows = [&](bf16* dst, int stride, int pieces, int from) {
        const int step = SD_THREADS / pieces, row0 = tid / pieces, c = tid % pieces * 8;
        if (row0 < step)
#pragma unroll 4
            for (int row = row0; row < G * KT; row += step) {
                const long long off = key_off[row % KT];
                sd_copy(dst + row * stride + c, off >= 0 ? a.pages + off + (row / KT) * head_step + from + c : a.pages, off >= 0);
            }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    __syncthreads();
    copy_rows(Ks, KS, qv, 0);                                    // group: the queries and the first keys
    copy_rows(Vs, VS, vv, D);
    const float to_cap = a.cap > 0.f ? a.scale / a.cap : 0.f, slope = -SD_LOG2_E * (a.cap > 0.f ? a.cap : a.scale);
    float o[SD_PIECES][2][4] = {};
    const int pieces = G * (DV / 16);
    for (int j0 = lo; j0 <= hi; j0 += KT) {
        const bool more = j0 + KT <= hi;
        const long long next = more && tid < KT ? place(j0 + KT + tid) : -1;
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                         // this tile's keys are in
        for (int unit = warp; unit < G * (KT / 8); unit += SD_WARPS) {
            const int group = unit % G, k0 = unit / G * 8;
            if (j0 + k0 > hi) {                                  // none of these keys is seen
                if (g < hpg) *reinterpret_cast<float2*>(Ws + (group * hpg + g) * PS + k0 + 2 * t) = make_float2(0.f, 0.f);
                if (g + 8 < hpg) *reinterpret_cast<float2*>(Ws + (group * hpg + g + 8) * PS + k0 + 2 * t) = make_float2(0.f, 0.f);
                continue;
            }
            float s0[4] = {}, s1[4] = {};
            const bf16* Qw = Qs + (group * 16 + (lane & 15)) * KS + (lane >> 4) * 8;
            const bf16* Kw = Ks + (group * KT + k0 + (lane & 7)) * KS + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int ks = 0; ks < D; ks += 32) {
                unsigned qa[4], b0, b1;
                sd_x4(qa, Qw + ks);
                sd_x2(b0, b1, Kw + ks);
                sd_mma(s0, qa, b0, b1);
                if (ks + 16 < D) {
                    sd_x4(qa, Qw + ks + 16);
                    sd_x2(b0, b1, Kw + ks + 16);
                    sd_mma(s1, qa, b0, b1);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (8 * r >= hpg) break;                         // (no such heads in any lane)
                const int h = group * hpg + min(g + 8 * r, hpg - 1);
                float w[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {                    // 1 / (1 + 2^(x slope - bias log2 e)), x the score or tanh(score to_cap)
                    float s = s0[2 * r + c] + s1[2 * r + c];
                    if (a.cap > 0.f) s = sd_tanh(s * to_cap);
                    w[c] = j0 + k0 + 2 * t + c <= hi ? sd_rcp(1.f + sd_ex2(fmaf(s, slope, bias[h]))) : 0.f;
                }
                if (g + 8 * r < hpg) *reinterpret_cast<float2*>(Ws + h * PS + k0 + 2 * t) = make_float2(w[0], w[1]);
            }
        }
        if (more && tid < KT) key_off[tid] = next;               // (this tile's copies were made of the places before)
        __syncthreads();                                         // the weights are in place, the keys and the places are free
        if (more) copy_rows(Ks, KS, qv, 0);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        {
            const int key = tid % KT;
            float w[SD_MAX_HEADS];
#pragma unroll
            for (int i = 0; i < SD_MAX_HEADS; ++i) w[i] = i < H ? Ws[i * PS + key] : 0.f;
            for (int h = tid / KT; h < H; h += SD_THREADS / KT) {
                float m = 0.f;
#pragma unroll
                for (int i = 0; i < SD_MAX_HEADS; ++i)
                    if (i < H) m = fmaf(mix[h * H + i], w[i], m);
                Ps[(h / hpg * 16 + h % hpg) * PS + key] = __float2bfloat16_rn(m);
            }
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");   // this tile's values are in
        __syncthreads();
        const int steps = (min(KT, hi - j0 + 1) + 15) / 16;      // 16 keys each; rows past the range are zeros
#pragma unroll
        for (int i = 0; i < SD_PIECES; ++i) {
            const int piece = warp + i * SD_WARPS;
            if (piece < pieces) {
                const int group = piece / (DV / 16), c0 = piece % (DV / 16) * 16;
                const bf16* Pw = Ps + (group * 16 + (lane & 15)) * PS + (lane >> 4) * 8;
                const bf16* Vw = Vs + (group * KT + (lane & 7) + ((lane >> 3) & 1) * 8) * VS + c0 + (lane >> 4) * 8;
#pragma unroll
                for (int k = 0; k < KT / 16; ++k) {
                    if (k >= steps) break;
                    unsigned pa[4], v[4];
                    sd_x4(pa, Pw + k * 16);
                    sd_x4_trans(v, Vw + k * 16 * VS);
                    sd_mma(o[i][0], pa, v[0], v[1]);
                    sd_mma(o[i][1], pa, v[2], v[3]);
                }
            }
        }
        if (more) {
            __syncthreads();                                     // the values and the mixed weights are free
            copy_rows(Vs, VS, vv, D);
        }
    }
#pragma unroll
    for (int i = 0; i < SD_PIECES; ++i) {
        const int piece = warp + i * SD_WARPS;
        if (piece >= pieces) continue;
        const int group = piece / (DV / 16), c0 = piece % (DV / 16) * 16 + 2 * t;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (g + 8 * r >= hpg) continue;
            const size_t col = (size_t)(group * hpg + g + 8 * r) * DV + c0;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float x = o[i][half][2 * r], y = o[i][half][2 * r + 1];
                if (a.partial) *reinterpret_cast<float2*>(a.partial + ((size_t)n * a.segments + blockIdx.y) * H * DV + col + 8 * half) = make_float2(x, y);
                else *reinterpret_cast<unsigned*>(a.out + (size_t)n * a.out_t + col + 8 * half) = sd_pack(x, y);
            }
        }
    }
}

// out[n, c] = the sum of partial[n, range, c] over the ranges that hold a key the token sees: warp w of a block adds ranges w, w + 8, ..,
// then the warps' sums are added in order; a lane has four columns.
constexpr int SD_SUM_WARPS = 8;
__global__ void __launch_bounds__(32 * SD_SUM_WARPS) sigmoid_decode_sum_kernel(const float* __restrict__ partial, const int* __restrict__ ctx_len,
                                                                         bf16* __restrict__ out, long out_t, int W, int segments, int segment_keys) {
    __shared__ float4 part[SD_SUM_WARPS][32];
    pdl_wait();                                    // what the kernels before wrote is complete
    pdl_trigger();
    const int n = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = (blockIdx.y * 32 + lane) * 4;
    const int used = min(segments, (ctx_len[n] - 1) / segment_keys + 1);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < W) {
        const float* at = partial + (size_t)n * segments * W + c;
#pragma unroll 4
        for (int k = warp; k < used; k += SD_SUM_WARPS) {
            const float4 v = *reinterpret_cast<const float4*>(at + (size_t)k * W);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp || c >= W) return;
#pragma unroll
    for (int w = 1; w < SD_SUM_WARPS; ++w) {
        const float4 v = part[w][lane];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    unsigned* o = reinterpret_cast<unsigned*>(out + (size_t)n * out_t + c);
    o[0] = sd_pack(s.x, s.y);
    o[1] = sd_pack(s.z, s.w);
}

constexpr size_t SD_MOST_BYTES = 220 * 1024;

template <int KT> void launch_decode(const SigDecodeArgs& a, int N, cudaStream_t stream) {
    const size_t smem = sd_smem(a.H, a.G, a.D, a.DV, KT);
#define LLMP_SD_CASE(A, B)                                                                                                     \
    if ((A == 0 || a.D == 16 * A) && (B == 0 || a.DV == 16 * B)) {                                                             \
        LLMP_ALLOW_SMEM((sigmoid_decode_kernel<KT, A, B>), smem);                                                              \
        llmp_launch_dependent(sigmoid_decode_kernel<KT, A, B>, dim3(N, a.segments), dim3(SD_THREADS), smem, stream, a);        \
    } else
    LLMP_SD_CASE(8, 8) LLMP_SD_CASE(4, 4) LLMP_SD_CASE(8, 4) LLMP_SD_CASE(4, 8) LLMP_SD_CASE(0, 0) {}
#undef LLMP_SD_CASE
}

}  // namespace

// sigmoid_attention_mma.cu
LLMP_API int llmp_sigmoid_attention_mma_supports(int H, int G, int d, int dv);

// Keys of a tile for these sizes (ranges are multiples of it), or 0: they are not served. The mixed weights are rounded to bfloat16 for
// the product with the values, so only sizes whose prompts have theirs rounded too; the general kernel keeps float32 for the others.
LLMP_API int llmp_sigmoid_decode_keys(int H, int G, int d, int dv) {
    if (!llmp_sigmoid_attention_mma_supports(H, G, d, dv) || H > SD_MAX_HEADS || G * (dv / 16) > SD_PIECES * SD_WARPS) return 0;
    for (int keys : {64, 32})
        if (sd_smem(H, G, d, dv, keys) <= SD_MOST_BYTES) return keys;
    return 0;
}

// One token a request: row n of the queries is request n's. partial: float32 [N, segments, H dv] where segments > 1, and segments *
// segment_keys the most keys a request may see.
LLMP_API int llmp_sigmoid_decode(const void* q, long q_t, const void* pages, const int* tables, int width, const int* ctx_len, const float* talk,
                                 const float* pb, void* out, long out_t, float* partial, int segments, int segment_keys, int N, int H, int G,
                                 int d, int dv, int page_size, float scale, float cap, cudaStream_t stream) {
    if (N <= 0) return 0;
    const int keys = llmp_sigmoid_decode_keys(H, G, d, dv);
    LLMP_REQUIRE(keys > 0, "sigmoid_decode: no kernel for heads=%d kv_heads=%d dim=%d vdim=%d", H, G, d, dv);
    LLMP_REQUIRE(page_size > 0 && width > 0 && q_t % 8 == 0 && out_t % 4 == 0 && ((size_t)q | (size_t)pages) % 16 == 0 && (size_t)out % 8 == 0,
                 "sigmoid_decode: page=%d width=%d, rows must be 16-byte aligned", page_size, width);
    LLMP_REQUIRE(segments >= 1 && segments <= 65535 && (segments == 1 || (partial && segment_keys > 0 && segment_keys % keys == 0)),
                 "sigmoid_decode: %d key ranges of %d keys", segments, segment_keys);
    SigDecodeArgs a;
    a.q = (const bf16*)q; a.q_t = q_t; a.pages = (const bf16*)pages; a.tables = tables; a.width = width; a.ctx_len = ctx_len; a.talk = talk;
    a.pb = pb; a.out = (bf16*)out; a.out_t = out_t; a.partial = segments > 1 ? partial : nullptr; a.H = H; a.G = G; a.D = d; a.DV = dv;
    a.page_size = page_size; a.segments = segments; a.segment_keys = segments > 1 ? segment_keys : 0; a.scale = scale; a.cap = cap;
    if (keys == 64) launch_decode<64>(a, N, stream);
    else launch_decode<32>(a, N, stream);
    if (segments > 1)
        llmp_launch_dependent(sigmoid_decode_sum_kernel, dim3(N, (H * dv + 127) / 128), dim3(32 * SD_SUM_WARPS), 0, stream, (const float*)partial, ctx_len,
                              (bf16*)out, out_t, H * dv, segments, segment_keys);
    return llmp_check_launch("sigmoid_decode");
}
