// The gated delta rule of delta_rule.cu for requests that bring a single token: everything between the layer's products in one kernel.
//
// A block takes a (request, head): the convolution of the head's query, key and value channels with its carried inputs, unit
// vectors, decays and beta, the step over the state
//   S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q = (diag(g) S)^T q + u (k . q)
// and the head's gated norm. As kernels of their own (convolution, preparation, walk, norm) these were four launches of which each
// waited for the one before, and the walk, whose blocks copy stages of eight tokens, took most of them: 8 requests of 16 heads of
// 128 x 128 28 us, 6 to 8 so; what bounds it is the state, 16.8 MB read and written (2.6 us at the copy rate), and the block's own chain
// of five phases. Everything is float32; the outputs are rounded once to the compute type. The state pieces are as short_conv.cu
// and delta_rule.cu keep them: two copies that take turns by the parity of the position.
//
// A warp holds whole rows of the state, 16 apart, a lane four columns of them, so all of the state is asked for in 16-byte
// words before the convolution begins.
#include "common.cuh"

namespace {

constexpr int DT_WARPS = 16, DT_THREADS = 32 * DT_WARPS;
constexpr int DT_MAX_TAPS = 8;

struct DeltaStepArgs {
    const float* proj; long proj_t;                        // [tokens, q | k | v | beta | ..] as projected
    const float* decay; long decay_t;                      // [tokens, H d], pre-activations
    const float* gate; long gate_t;                        // [tokens, H dv], before the sigmoid
    const float* taps;                                     // [C, K]
    const float* a_log; const float* dt_bias; const float* norm;      // [H], [H d], [dv]
    float* state; long state_slot; long conv_half; long scan_offset; long scan_half;
    const int* q_start; const int* slots; const int* positions;
    void* out; long out_t;
    int H, G, d, dv, K;
    float eps;
};

__device__ __forceinline__ float dt_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// NR: rows of the state a warp holds (16 NR >= d).
template <typename T, int NR>
__global__ void __launch_bounds__(DT_THREADS) delta_step_kernel(const DeltaStepArgs a) {
    extern __shared__ __align__(16) float dt_smem[];
    const int d = a.d, dv = a.dv, K = a.K;
    float* const qs = dt_smem;                             // [d]
    float* const ks = qs + d;                              // [d]
    float* const gs = ks + d;                              // [d]
    float* const vs = gs + d;                              // [dv]
    float* const part = vs + dv;                           // [DT_WARPS][2 dv]: a warp's shares of S^T k | S^T q
    float* const sums = part + DT_WARPS * 2 * dv;          // [2 dv]: u | S^T q
    const int h = blockIdx.y, r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = a.H / a.G, kh = h / group, C = 2 * a.G * d + a.H * dv;
    // the channel that a thread filters
    const int c = tid < d ? kh * d + tid : (tid < 2 * d ? a.G * d + kh * d + tid - d : 2 * a.G * d + h * dv + tid - 2 * d);
    const bool filters = tid < 2 * d + dv;
    float tap[DT_MAX_TAPS];                                // weights: nothing of the step writes them
#pragma unroll
    for (int j = 0; j < DT_MAX_TAPS; ++j) tap[j] = filters && j < K ? a.taps[(size_t)c * K + j] : 0.f;
    const float rate = tid < d ? -expf(a.a_log[h]) : 0.f, dt_b = tid < d ? a.dt_bias[(size_t)h * d + tid] : 0.f;
    pdl_wait();                                            // what the kernels before wrote is complete
    pdl_trigger();
    const int t = a.q_start[r];
    if (a.q_start[r + 1] - t != 1) return;
    const int p = a.positions[t];
    float* slot = a.state + (size_t)a.slots[r] * a.state_slot;
    const int rd = (p + 1) & 1, wr = p & 1;
    const size_t head = (size_t)a.scan_offset + (size_t)h * d * dv + lane * 4;
    const float* from = slot + head + rd * a.scan_half;
    const bool mine = lane * 4 < dv;
    float4 S[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int row = i * DT_WARPS + warp;
        S[i] = mine && row < d ? *reinterpret_cast<const float4*>(from + (size_t)row * dv) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float beta = 1.f / (1.f + expf(-a.proj[(size_t)t * a.proj_t + C + h]));
    if (filters) {
        const float* before = slot + rd * a.conv_half + c;
        float* after = slot + wr * a.conv_half + c;
        const bool keeps = tid >= 2 * d || h % group == 0;     // of the heads that share a query/key head the first leaves its inputs
        const float x = a.proj[(size_t)t * a.proj_t + c];
        float acc = 0.f, last = 0.f;
#pragma unroll
        for (int j = 0; j < DT_MAX_TAPS; ++j) {
            if (j < K - 1) {
                const float w = before[(size_t)j * C];
                acc = fmaf(w, tap[j], acc);
                if (j > 0 && keeps) after[(size_t)(j - 1) * C] = w;
            } else if (j == K - 1) {
                last = tap[j];
            }
        }
        acc = fmaf(x, last, acc);
        if (K > 1 && keeps) after[(size_t)(K - 2) * C] = x;
        const float y = acc / (1.f + expf(-acc));
        if (tid < d) qs[tid] = y;
        else if (tid < 2 * d) ks[tid - d] = y;
        else vs[tid - 2 * d] = y;
    }
    if (tid < d) gs[tid] = expf(rate * dt_softplus(a.decay[(size_t)t * a.decay_t + (size_t)h * d + tid] + dt_b));
    __syncthreads();
    float kk = 0.f, qq = 0.f, kq = 0.f;                    // every warp for itself
    for (int i = lane; i < d; i += 32) {
        kk = fmaf(ks[i], ks[i], kk);
        qq = fmaf(qs[i], qs[i], qq);
        kq = fmaf(ks[i], qs[i], kq);
    }
    kk = warp_sum(kk);
    qq = warp_sum(qq);
    kq = warp_sum(kq);
    const float kf = 1.f / sqrtf(kk + 1e-6f), qf = (1.f / sqrtf((float)d)) / sqrtf(qq + 1e-6f);
    float4 sk = make_float4(0.f, 0.f, 0.f, 0.f), sq = sk;
    float kn[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int row = i * DT_WARPS + warp;
        const bool have = row < d;
        const float g = have ? gs[row] : 0.f, q = have ? qs[row] * qf : 0.f;
        kn[i] = have ? ks[row] * kf : 0.f;
        S[i] = make_float4(S[i].x * g, S[i].y * g, S[i].z * g, S[i].w * g);
        sk = make_float4(fmaf(S[i].x, kn[i], sk.x), fmaf(S[i].y, kn[i], sk.y), fmaf(S[i].z, kn[i], sk.z), fmaf(S[i].w, kn[i], sk.w));
        sq = make_float4(fmaf(S[i].x, q, sq.x), fmaf(S[i].y, q, sq.y), fmaf(S[i].z, q, sq.z), fmaf(S[i].w, q, sq.w));
    }
    if (mine) {
        reinterpret_cast<float4*>(part + warp * 2 * dv)[lane] = sk;
        reinterpret_cast<float4*>(part + warp * 2 * dv + dv)[lane] = sq;
    }
    __syncthreads();
    if (tid < 2 * dv) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < DT_WARPS; ++w) s += part[w * 2 * dv + tid];
        sums[tid] = tid < dv ? beta * (vs[tid] - s) : s;
    }
    __syncthreads();
    const float4 u = mine ? reinterpret_cast<const float4*>(sums)[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp == 0) {                                       // the head's outputs
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f), z = o, w = o;
        if (mine) {
            const float4 s = reinterpret_cast<const float4*>(sums + dv)[lane];
            const float both = kq * kf * qf;
            o = make_float4(fmaf(u.x, both, s.x), fmaf(u.y, both, s.y), fmaf(u.z, both, s.z), fmaf(u.w, both, s.w));
            const float* gate = a.gate + (size_t)t * a.gate_t + (size_t)h * dv + lane * 4;
            z = make_float4(gate[0], gate[1], gate[2], gate[3]);
            w = make_float4(a.norm[lane * 4], a.norm[lane * 4 + 1], a.norm[lane * 4 + 2], a.norm[lane * 4 + 3]);
        }
        const float ss = warp_sum(fmaf(o.x, o.x, fmaf(o.y, o.y, fmaf(o.z, o.z, o.w * o.w))));
        const float inv = 1.f / sqrtf(ss / (float)dv + a.eps);
        if (mine) {
            T* out = reinterpret_cast<T*>(a.out) + (size_t)t * a.out_t + (size_t)h * dv + lane * 4;
            out[0] = from_float<T>(o.x * inv * w.x / (1.f + expf(-z.x)));
            out[1] = from_float<T>(o.y * inv * w.y / (1.f + expf(-z.y)));
            out[2] = from_float<T>(o.z * inv * w.z / (1.f + expf(-z.z)));
            out[3] = from_float<T>(o.w * inv * w.w / (1.f + expf(-z.w)));
        }
    }
    float* to = slot + head + wr * a.scan_half;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int row = i * DT_WARPS + warp;
        if (mine && row < d)
            *reinterpret_cast<float4*>(to + (size_t)row * dv) = make_float4(fmaf(kn[i], u.x, S[i].x), fmaf(kn[i], u.y, S[i].y),
                                                                           fmaf(kn[i], u.z, S[i].z), fmaf(kn[i], u.w, S[i].w));
    }
}

template <typename T> void launch_step(const DeltaStepArgs& a, int R, cudaStream_t stream) {
    const size_t smem = (size_t)(3 * a.d + a.dv + (DT_WARPS + 1) * 2 * a.dv) * sizeof(float);
    auto launch = [&](auto kernel) { llmp_launch_dependent(kernel, dim3(R, a.H), dim3(DT_THREADS), smem, stream, a); };
    if (a.d <= DT_WARPS) launch(delta_step_kernel<T, 1>);
    else if (a.d <= 2 * DT_WARPS) launch(delta_step_kernel<T, 2>);
    else if (a.d <= 4 * DT_WARPS) launch(delta_step_kernel<T, 4>);
    else if (a.d <= 8 * DT_WARPS) launch(delta_step_kernel<T, 8>);
    else launch(delta_step_kernel<T, 12>);
}

}  // namespace

// Heads that a block's threads can hold: a thread a filtered channel, a lane four columns; all offsets into the state in 16-byte steps.
LLMP_API int llmp_delta_step_serves(int channels, int d, int dv, int K) {
    return d > 0 && dv > 0 && d % 4 == 0 && dv % 4 == 0 && dv <= 128 && d <= 12 * DT_WARPS && 2 * d + dv <= DT_THREADS && K >= 1 && K <= DT_MAX_TAPS &&
           (long)2 * (K - 1) * channels % 4 == 0;
}

// Requests of a single token; the others are left alone. state: the slot's two pieces, [2][K - 1][C] inputs of the convolution at the
// front and [2][H][d][dv] at scan_offset.
LLMP_API int llmp_delta_step(const float* proj, long proj_t, const float* decay, long decay_t, const float* gate, long gate_t,
                             const float* taps, const float* a_log, const float* dt_bias, const float* norm, float* state, long state_slot,
                             long scan_offset, const int* q_start, const int* slots, const int* positions, void* out, int out_dtype,
                             long out_t, int R, int H, int G, int d, int dv, int K, float eps, cudaStream_t stream) {
    if (R <= 0) return 0;
    LLMP_REQUIRE(H > 0 && G > 0 && H % G == 0 && H <= 65535, "delta_step: bad sizes heads=%d qk_heads=%d", H, G);
    const int C = 2 * G * d + H * dv;
    LLMP_REQUIRE(llmp_delta_step_serves(C, d, dv, K), "delta_step: heads of %d x %d with %d taps are not served", d, dv, K);
    LLMP_REQUIRE((size_t)state % 16 == 0 && state_slot % 4 == 0 && scan_offset >= (long)2 * (K - 1) * C && scan_offset % 4 == 0,
                 "delta_step: the state's pieces overlap or are not 16-byte aligned");
    DeltaStepArgs a;
    a.proj = proj; a.proj_t = proj_t; a.decay = decay; a.decay_t = decay_t; a.gate = gate; a.gate_t = gate_t; a.taps = taps; a.a_log = a_log;
    a.dt_bias = dt_bias; a.norm = norm; a.state = state; a.state_slot = state_slot; a.conv_half = (long)(K - 1) * C; a.scan_offset = scan_offset;
    a.scan_half = (long)H * d * dv; a.q_start = q_start; a.slots = slots; a.positions = positions; a.out = out; a.out_t = out_t; a.H = H; a.G = G;
    a.d = d; a.dv = dv; a.K = K; a.eps = eps;
    if (out_dtype == LLMP_BF16) launch_step<bf16>(a, R, stream);
    else launch_step<float>(a, R, stream);
    return llmp_check_launch("delta_step");
}
