// Latent attention of single tokens (bfloat16, mma.sync, float32 sums), with the cache and the results of latent_attention_mma.cu.
//
// A decoded token's rows are its heads: 16 of them are one m16 tile, which the tile of 64 rows there fills a quarter of, two of eight
// warps at work. Here a block takes up to 16 heads of one token and one range of keys, 128 keys at a time, whose rows come in
// two halves of 64 by 16-byte cp.async, all asked for at once. Scores: a warp makes those of 8 keys of each half over the whole row.
// Softmax: the warps' maxima and sums meet in shared memory, the probabilities go there as two bfloat16 halves. (One half was 0.6 %
// further from 64 bits than latent_attention_mma on average, whose smaller key tiles leave more probabilities at exactly 1; with two
// 2.8 % nearer, at no cost: the products share the values' fragments.) Values: a warp makes an
// eighth of the latent's columns over all 128 keys, which lie in shared memory already. A range of more keys goes on with a
// running softmax. With several ranges the blocks leave unnormalised sums, and a second kernel adds a row's in ascending order.
// 8 requests of 2,048 keys, 16 heads, latents of 512 + 64: 37 us there (ranges of 256 keys), 22 here (as single launches; a layer of
// one graph 71 us there, 53 here).
#include "common.cuh"

namespace {

constexpr int LD_KEYS = 128, LD_HALF = 64, LD_THREADS = 256, LD_ROWS = 16;
constexpr int LD_PS = LD_KEYS + 8;

struct LatentDecodeArgs {
    const bf16* q_lat; long ql_t, ql_h;
    const bf16* q_rot; long qr_t, qr_h;
    bf16* out; long o_t, o_h;
    const bf16* pages;
    const int* tables; int table_stride;
    const int* ctx_len;
    float* part_o; float* part_ml;          // null: one range, the result goes to `out`
    const float* sink;
    int N, H, rot, page_size, range_keys;
    float scale;
};

__device__ __forceinline__ void ld_cp_async_16(void* smem_dst, const void* gmem_src, bool valid) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem_src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ld_x4(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_x4_trans(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_x2(unsigned& r0, unsigned& r1, const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ld_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned ld_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

// C128: the latent's size / 128.
template <int C128>
__global__ void __launch_bounds__(LD_THREADS, 1) latent_decode_kernel(const LatentDecodeArgs a) {
    extern __shared__ __align__(16) unsigned char ld_raw[];
    constexpr int RANK = C128 * 128, NT = C128 * 2;              // n8 tiles of a warp's columns
    const int dk = RANK + a.rot, stride = dk + 8, pieces = dk / 8;
    bf16* Qs = reinterpret_cast<bf16*>(ld_raw);                  // [16][stride]
    bf16* Ks = Qs + LD_ROWS * stride;                            // [128][stride]: keys, and in their first columns values
    bf16* Ps = Ks + (size_t)LD_KEYS * stride;                    // [16][LD_PS]: probabilities, then what their rounding left
    bf16* Pl = Ps + LD_ROWS * LD_PS;
    __shared__ float row_max[8][LD_ROWS], row_sum[8][LD_ROWS];
    __shared__ long long key_off[LD_KEYS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int n = blockIdx.x, head0 = blockIdx.y * LD_ROWS, heads = min(LD_ROWS, a.H - head0);
    pdl_trigger();
    pdl_wait();
    const int last = a.ctx_len[n] - 1;                           // the token's own key
    const int lo = blockIdx.z * a.range_keys, hi = a.part_o ? min(last, lo + a.range_keys - 1) : last;
    if (lo > hi) return;                                         // the token does not see this range; the merge knows
    const int* table = a.tables + (size_t)n * a.table_stride;

    for (int e = tid; e < LD_ROWS * pieces; e += LD_THREADS) {
        const int row = e / pieces, c = (e % pieces) * 8;
        const bool ok = row < heads;
        const bf16* src = a.q_lat;
        if (ok) src = c < RANK ? a.q_lat + (size_t)n * a.ql_t + (size_t)(head0 + row) * a.ql_h + c
                               : a.q_rot + (size_t)n * a.qr_t + (size_t)(head0 + row) * a.qr_h + (c - RANK);
        ld_cp_async_16(Qs + row * stride + c, src, ok);
    }
    float o[NT][4] = {}, m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    const float scale_log2 = a.scale * 1.4426950408889634f;
    for (int j0 = lo; j0 <= hi; j0 += LD_KEYS) {
        if (tid < LD_KEYS) {
            const int j = j0 + tid;
            long long off = -1;
            if (j <= hi) {
                const int page = table[j / a.page_size];
                if (page >= 0) off = (long long)((size_t)page * a.page_size + j % a.page_size) * dk;
            }
            key_off[tid] = off;
        }
        __syncthreads();                                         // also: everyone has left the keys of the round before
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            for (int e = tid; e < LD_HALF * pieces; e += LD_THREADS) {
                const int key = half * LD_HALF + e / pieces, c = (e % pieces) * 8;
                const long long off = key_off[key];
                ld_cp_async_16(Ks + (size_t)key * stride + c, off >= 0 ? a.pages + off + c : a.pages, off >= 0);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        float s[2][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (half == 0) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();
            float acc[4][4] = {};                                // four chains: the products of a single one would wait for each other
            const bf16* Kw = Ks + (size_t)(half * LD_HALF + warp * 8 + (lane & 7)) * stride + ((lane >> 3) & 1) * 8;
            const bf16* Qw = Qs + (lane & 15) * stride + (lane >> 4) * 8;
            for (int k0 = 0; k0 < dk / 16; k0 += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int ks = k0 + u;
                    if (ks >= dk / 16) break;
                    unsigned qa[4], b0, b1;
                    ld_x4(qa, Qw + ks * 16);
                    ld_x2(b0, b1, Kw + ks * 16);
                    ld_mma(acc[u], qa, b0, b1);
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[half][c] = ((acc[0][c] + acc[1][c]) + (acc[2][c] + acc[3][c])) * scale_log2;
                if (j0 + half * LD_HALF + warp * 8 + 2 * t + (c & 1) > hi) s[half][c] = -INFINITY;
            }
        }
        float mx[2], m_new[2], alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r] = fmaxf(fmaxf(s[0][2 * r], s[0][2 * r + 1]), fmaxf(s[1][2 * r], s[1][2 * r + 1]));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            if (t == 0) row_max[warp][g + 8 * r] = mx[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float m = m_run[r];
#pragma unroll
            for (int w = 0; w < 8; ++w) m = fmaxf(m, row_max[w][g + 8 * r]);
            m_new[r] = m;
            alpha[r] = m > -INFINITY ? ld_ex2(m_run[r] - m) : 1.f;
            m_run[r] = m;
            const float base = m > -INFINITY ? m : 0.f;
            float sum = 0.f;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float p0 = ld_ex2(s[half][2 * r] - base), p1 = ld_ex2(s[half][2 * r + 1] - base);
                sum += p0 + p1;
                const unsigned hi2 = ld_pack(p0, p1);
                const int at = (g + 8 * r) * LD_PS + half * LD_HALF + warp * 8 + 2 * t;
                *reinterpret_cast<unsigned*>(Ps + at) = hi2;
                *reinterpret_cast<unsigned*>(Pl + at) = ld_pack(p0 - __uint_as_float(hi2 << 16), p1 - __uint_as_float(hi2 & 0xffff0000u));
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if (t == 0) row_sum[warp][g + 8 * r] = sum;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) sum += row_sum[w][g + 8 * r];
            l_run[r] = l_run[r] * alpha[r] + sum;
        }
        if (j0 > lo) {
#pragma unroll
            for (int i = 0; i < NT; ++i) { o[i][0] *= alpha[0]; o[i][1] *= alpha[0]; o[i][2] *= alpha[1]; o[i][3] *= alpha[1]; }
        }
        const int steps = min(LD_KEYS, hi - j0 + 16) / 16;       // 16 keys each; rows past the range are zeros
        for (int k = 0; k < steps; ++k) {
            unsigned pa[4], pl[4];
            ld_x4(pa, Ps + (lane & 15) * LD_PS + k * 16 + (lane >> 4) * 8);
            ld_x4(pl, Pl + (lane & 15) * LD_PS + k * 16 + (lane >> 4) * 8);
            const bf16* Vw = Ks + (size_t)(k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * stride + warp * NT * 8 + (lane >> 4) * 8;
#pragma unroll
            for (int i = 0; i < NT; i += 2) {
                unsigned v[4];
                ld_x4_trans(v, Vw + i * 8);
                ld_mma(o[i], pa, v[0], v[1]);
                ld_mma(o[i + 1], pa, v[2], v[3]);
                ld_mma(o[i], pl, v[0], v[1]);
                ld_mma(o[i + 1], pl, v[2], v[3]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = g + 8 * r;
        if (row >= heads) continue;
        const int col = warp * NT * 8 + 2 * t;
        if (a.part_o) {
            const size_t at = ((size_t)blockIdx.z * a.N + n) * a.H + head0 + row;
            float* dst = a.part_o + at * RANK + col;
#pragma unroll
            for (int i = 0; i < NT; ++i) *reinterpret_cast<float2*>(dst + i * 8) = make_float2(o[i][2 * r], o[i][2 * r + 1]);
            if (warp == 0 && t == 0) {
                a.part_ml[at * 2] = m_run[r];
                a.part_ml[at * 2 + 1] = l_run[r];
            }
        } else {
            float inv = l_run[r] > 0.f ? 1.f / l_run[r] : 0.f;
            if (a.sink) {                                        // a key of score sink[h] without a value
                const float sk = a.sink[head0 + row] * 1.4426950408889634f;
                const float m = fmaxf(m_run[r], sk);
                const float w = m_run[r] > -INFINITY ? ld_ex2(m_run[r] - m) : 0.f;
                inv = w / (l_run[r] * w + ld_ex2(sk - m));
            }
            bf16* dst = a.out + (size_t)n * a.o_t + (size_t)(head0 + row) * a.o_h + col;
#pragma unroll
            for (int i = 0; i < NT; ++i) *reinterpret_cast<unsigned*>(dst + i * 8) = ld_pack(o[i][2 * r] * inv, o[i][2 * r + 1] * inv);
        }
    }
}

// out = sum_s 2^(m_s - m) o_s / sum_s 2^(m_s - m) l_s over the ranges that hold keys the token sees, in ascending order. A block per
// (token, head), four columns a thread. The first LD_MERGE_AHEAD ranges' sums are asked for beside the maxima and the sums of weights
// (one load after another took 6.0 us of a decoding layer's 53).
constexpr int LD_MAX_RANGES = 1024, LD_MERGE_AHEAD = 16;
__global__ void __launch_bounds__(128) latent_decode_merge_kernel(const LatentDecodeArgs a, int rank) {
    __shared__ float weight[LD_MAX_RANGES], part[8];
    const int n = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    pdl_trigger();
    pdl_wait();
    const int ranges = (a.ctx_len[n] - 1) / a.range_keys + 1;
    const size_t step = (size_t)a.N * a.H, first = (size_t)n * a.H + h;
    const float* from = a.part_o + first * rank + tid * 4;
    float4 v[LD_MERGE_AHEAD];
#pragma unroll
    for (int s = 0; s < LD_MERGE_AHEAD; ++s)
        v[s] = s < ranges && tid * 4 < rank ? *reinterpret_cast<const float4*>(from + s * step * rank) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float sk = a.sink ? a.sink[h] * 1.4426950408889634f : -INFINITY;
    float m = sk, l = 0.f;
    const float2 own = tid < ranges ? *reinterpret_cast<const float2*>(a.part_ml + (tid * step + first) * 2) : make_float2(-INFINITY, 0.f);
    m = fmaxf(m, own.x);
    for (int s = tid + 128; s < ranges; s += 128) m = fmaxf(m, a.part_ml[(s * step + first) * 2]);
    m = warp_max(m);
    if ((tid & 31) == 0) part[tid >> 5] = m;
    __syncthreads();
    m = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
    if (tid < ranges) {
        weight[tid] = m > -INFINITY ? ld_ex2(own.x - m) : 0.f;
        l = weight[tid] * own.y;
    }
    for (int s = tid + 128; s < ranges; s += 128) {
        const float2 other = *reinterpret_cast<const float2*>(a.part_ml + (s * step + first) * 2);
        weight[s] = m > -INFINITY ? ld_ex2(other.x - m) : 0.f;
        l = fmaf(weight[s], other.y, l);
    }
    l = warp_sum(l);
    if ((tid & 31) == 0) part[4 + (tid >> 5)] = l;
    __syncthreads();
    l = ((part[4] + part[5]) + (part[6] + part[7])) + (a.sink ? ld_ex2(sk - m) : 0.f);
    const float inv = l > 0.f ? 1.f / l : 0.f;
    if (tid * 4 >= rank) return;                                 // (the latent has up to 512 columns: four a thread)
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 0; s < LD_MERGE_AHEAD; ++s) {
        const float w = s < ranges ? weight[s] : 0.f;
        acc.x = fmaf(w, v[s].x, acc.x); acc.y = fmaf(w, v[s].y, acc.y); acc.z = fmaf(w, v[s].z, acc.z); acc.w = fmaf(w, v[s].w, acc.w);
    }
#pragma unroll 8
    for (int s = LD_MERGE_AHEAD; s < ranges; ++s) {
        const float4 u = *reinterpret_cast<const float4*>(from + s * step * rank);
        const float w = weight[s];
        acc.x = fmaf(w, u.x, acc.x); acc.y = fmaf(w, u.y, acc.y); acc.z = fmaf(w, u.z, acc.z); acc.w = fmaf(w, u.w, acc.w);
    }
    unsigned* o = reinterpret_cast<unsigned*>(a.out + (size_t)n * a.o_t + (size_t)h * a.o_h + tid * 4);
    o[0] = ld_pack(acc.x * inv, acc.y * inv);
    o[1] = ld_pack(acc.z * inv, acc.w * inv);
}

size_t ld_smem(int rank, int rot) { return sizeof(bf16) * ((size_t)(LD_ROWS + LD_KEYS) * (rank + rot + 8) + 2 * LD_ROWS * LD_PS); }

template <int C128> void launch_decode(const LatentDecodeArgs& a, int ranges, cudaStream_t stream) {
    const size_t smem = ld_smem(C128 * 128, a.rot);
    LLMP_ALLOW_SMEM(latent_decode_kernel<C128>, smem);
    llmp_launch_dependent(latent_decode_kernel<C128>, dim3(a.N, (a.H + LD_ROWS - 1) / LD_ROWS, ranges), dim3(LD_THREADS), smem, stream, a);
}

}  // namespace

LLMP_API int llmp_latent_decode_supports(int rank, int rot, int page_size) {
    return rank > 0 && rank % 128 == 0 && rank <= 512 && rot >= 0 && rot % 16 == 0 && page_size > 0 && ld_smem(rank, rot) <= 220 * 1024;
}

// One token a request: row n of the queries is request n's. scratch: float32, ranges * N * H * (rank + 2) entries where ranges > 1,
// ranges * range_keys the most keys a request may see.
LLMP_API int llmp_latent_decode(const void* q_lat, long ql_t, long ql_h, const void* q_rot, long qr_t, long qr_h, const void* pages,
                                const int* tables, int table_stride, const int* ctx_len, void* out, long o_t, long o_h, int N, int H, int rank,
                                int rot, int page_size, float scale, int range_keys, int ranges, float* scratch, const float* sink,
                                cudaStream_t stream) {
    if (N <= 0) return 0;
    LLMP_REQUIRE(llmp_latent_decode_supports(rank, rot, page_size), "latent_decode: sizes rank=%d rot=%d are not served", rank, rot);
    LLMP_REQUIRE(ql_t % 8 == 0 && ql_h % 8 == 0 && qr_t % 8 == 0 && qr_h % 8 == 0 && o_t % 2 == 0 && o_h % 2 == 0 && (size_t)q_lat % 16 == 0 &&
                 (size_t)q_rot % 16 == 0 && (size_t)out % 4 == 0 && (size_t)pages % 16 == 0, "latent_decode: query rows must be 16-byte aligned");
    LLMP_REQUIRE(ranges >= 1 && ranges <= LD_MAX_RANGES && (ranges == 1 || (scratch && range_keys > 0 && range_keys % LD_KEYS == 0)),
                 "latent_decode: %d ranges of %d keys", ranges, range_keys);
    LLMP_REQUIRE(H > 0 && (H + LD_ROWS - 1) / LD_ROWS <= 65535, "latent_decode: %d heads", H);
    LatentDecodeArgs a;
    a.q_lat = (const bf16*)q_lat; a.ql_t = ql_t; a.ql_h = ql_h; a.q_rot = (const bf16*)q_rot; a.qr_t = qr_t; a.qr_h = qr_h;
    a.out = (bf16*)out; a.o_t = o_t; a.o_h = o_h; a.pages = (const bf16*)pages; a.tables = tables; a.table_stride = table_stride;
    a.ctx_len = ctx_len; a.part_o = ranges > 1 ? scratch : nullptr;
    a.part_ml = ranges > 1 ? scratch + (size_t)ranges * N * H * rank : nullptr;
    a.sink = sink; a.N = N; a.H = H; a.rot = rot; a.page_size = page_size; a.range_keys = ranges > 1 ? range_keys : 0; a.scale = scale;
    if (rank == 128) launch_decode<1>(a, ranges, stream);
    else if (rank == 256) launch_decode<2>(a, ranges, stream);
    else if (rank == 384) launch_decode<3>(a, ranges, stream);
    else launch_decode<4>(a, ranges, stream);
    if (ranges > 1) llmp_launch_dependent(latent_decode_merge_kernel, dim3(N, H), dim3(128), 0, stream, a, rank);
    return llmp_check_launch("latent_decode");
}
