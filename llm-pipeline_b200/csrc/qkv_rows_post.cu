// Between a layer's float32 product [q | k | v] and its attention, in 16-byte pieces: bias, rotation of the first `rot` entries of every
// query and key head (entry i with i + rot / 2), a root mean square norm of every value head, queries to their rows and keys and values to
// the token's page slot, in the compute type. The row steps of sigmoid_attention.cu and capped_attention.cu, which keep rows that
// are not aligned.
//
// A warp takes 128 neighbouring entries of a token's queries and keys, or one value head, a lane four entries, so that the few rows of a
// decode step are one load deep: with a block a token and an entry a thread 16 rows of 3,072 entries took 6.5 us of a decoding layer,
// 2.2 so, and 2,048 rows with rotation 20 us, 17 so (37.7 MB, 5.8 us at the copy rate; four tokens a warp, all asked for at once: 17).
#include "common.cuh"

namespace {

constexpr int RP_WARPS = 4, RP_MAX_VALUE_PIECES = 4;

struct RowsArgs {
    const float* qkv; long qkv_t;
    const void* bias; int bias_bf16;
    const float* cos_t; const float* sin_t; int rot;
    float v_eps; int v_norm;
    void* q_out; long q_out_t;
    const int* slots; void* pages;
    int page_size, H, G, d, dv;
};

__device__ __forceinline__ float4 rp_load(const RowsArgs& a, const float* row, int at) {          // with its bias
    float4 v = *reinterpret_cast<const float4*>(row + at);
    if (!a.bias) return v;
    if (a.bias_bf16) {
        const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(a.bias) + at);
        const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        return make_float4(v.x + __low2float(lo), v.y + __high2float(lo), v.z + __low2float(hi), v.w + __high2float(hi));
    }
    const float4 b = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.bias) + at);
    return make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
}
__device__ __forceinline__ void rp_store(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void rp_store(bf16* p, const float4& v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
}

template <typename T>
__global__ void __launch_bounds__(32 * RP_WARPS) qkv_rows_post_kernel(const RowsArgs a) {
    pdl_wait();                                    // what the kernels before wrote is complete
    pdl_trigger();
    const int n = blockIdx.y, lane = threadIdx.x & 31, unit = blockIdx.x * RP_WARPS + (threadIdx.x >> 5);
    const int heads = (a.H + a.G) * a.d, head_units = (heads + 127) / 128;
    const float* row = a.qkv + (size_t)n * a.qkv_t;
    const int rs = a.d + a.dv;
    T* page_row = nullptr;
    if (a.pages && a.slots) {
        const int slot = a.slots[n];
        if (slot >= 0) page_row = reinterpret_cast<T*>(a.pages) + (((size_t)(slot / a.page_size) * a.G) * a.page_size + slot % a.page_size) * rs;
    }
    const size_t head_stride = (size_t)a.page_size * rs;
    if (unit < head_units) {
        const int at = unit * 128 + lane * 4;
        if (at >= heads) return;
        const int head = at / a.d, c = at % a.d;
        float4 v = rp_load(a, row, at);
        if (c < a.rot) {
            const int half = a.rot >> 1;
            const bool first = c < half;
            const int f = first ? c : c - half;
            const float4 o = rp_load(a, row, first ? at + half : at - half);
            const float4 cs = *reinterpret_cast<const float4*>(a.cos_t + (size_t)n * half + f), sn = *reinterpret_cast<const float4*>(a.sin_t + (size_t)n * half + f);
            const float s = first ? -1.f : 1.f;
            v = make_float4(v.x * cs.x + s * (o.x * sn.x), v.y * cs.y + s * (o.y * sn.y), v.z * cs.z + s * (o.z * sn.z), v.w * cs.w + s * (o.w * sn.w));
        }
        if (head < a.H) rp_store(reinterpret_cast<T*>(a.q_out) + (size_t)n * a.q_out_t + at, v);
        else if (page_row) rp_store(page_row + (size_t)(head - a.H) * head_stride + c, v);
        return;
    }
    const int g = unit - head_units;
    if (g >= a.G || !page_row) return;
    float4 v[RP_MAX_VALUE_PIECES];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < RP_MAX_VALUE_PIECES; ++i) {
        const int c = i * 128 + lane * 4;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < a.dv) v[i] = rp_load(a, row, heads + g * a.dv + c);
        ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
    }
    const float f = a.v_norm ? 1.f / sqrtf(warp_sum(ss) / (float)a.dv + a.v_eps) : 1.f;
    T* to = page_row + (size_t)g * head_stride + a.d;
#pragma unroll
    for (int i = 0; i < RP_MAX_VALUE_PIECES; ++i) {
        const int c = i * 128 + lane * 4;
        if (c < a.dv) rp_store(to + c, make_float4(v[i].x * f, v[i].y * f, v[i].z * f, v[i].w * f));
    }
}

}  // namespace

// 0: launched; 1: these rows are not aligned, the caller's own kernel takes them.
LLMP_API int llmp_qkv_rows_post(const float* qkv, long qkv_t, const void* bias, int bias_bf16, const float* cos_t, const float* sin_t, int rot,
                                float v_eps, int v_norm, void* q_out, int dtype, long q_out_t, const int* slots, void* pages, int page_size, int N,
                                int H, int G, int d, int dv, cudaStream_t stream) {
    if (d % 4 || dv % 4 || dv > 128 * RP_MAX_VALUE_PIECES || rot % 8 || qkv_t % 4 || q_out_t % 4 || N > 65535) return 1;
    if (((size_t)qkv | (size_t)cos_t | (size_t)sin_t | (size_t)q_out | (size_t)pages) % 16 || (size_t)bias % (bias_bf16 ? 8 : 16)) return 1;
    const RowsArgs a = {qkv, qkv_t, bias, bias_bf16, cos_t, sin_t, rot, v_eps, v_norm, q_out, q_out_t, slots, pages, page_size, H, G, d, dv};
    const int units = ((H + G) * d + 127) / 128 + (pages && slots ? G : 0);
    const dim3 grid((unsigned)((units + RP_WARPS - 1) / RP_WARPS), N);
    if (dtype == LLMP_F32) llmp_launch_dependent(qkv_rows_post_kernel<float>, grid, dim3(32 * RP_WARPS), 0, stream, a);
    else llmp_launch_dependent(qkv_rows_post_kernel<bf16>, grid, dim3(32 * RP_WARPS), 0, stream, a);
    return 0;
}
