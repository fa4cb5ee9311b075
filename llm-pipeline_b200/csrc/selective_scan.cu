// The selective state-space recurrence with a decay per channel and state entry.
//
// For every channel c of `inner` and state entry n of `states`, token by token:
//   dt_c = softplus(dt_raw_c + dt_bias_c)
//   S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n          (A < 0 comes from the caller; S is zero before the first token)
//   y_c = sum_n S[c, n] C_n + D_c x_c;      out_c = y_c * silu(z_c)   (without z: y_c)
// x (after its convolution and activation), dt_raw, B, C and z are float32 rows of the step; everything here is float32
// where the output is bfloat16. Where the output is float32 (the engine's true 32-bit path) the decays, the state and the
// read-out of a step are float64 between the float32 state a step reads and the one it leaves: a float32 recurrence over a
// thousand tokens with decays near one drifts by tens of units in the last place, which this keeps out of the sharper path.
// out has the compute type. Between steps a request keeps S in its state slot, as two copies [inner][states] that take
// turns by the parity of the last position written, so a step of one token never overwrites what it read.
//
// Two forms. Steps whose longest portion is long (the caller's rule: above 288 tokens), where the output is bfloat16 and a channel has
// up to 32 state entries: segments of SEG_TOKENS tokens side by side, for all requests of the step (below, at `SegArgs`). Else,
// token by token: a block is one warp and takes 32 / L
// channels of one request: L lanes share a channel and hold NS state entries each (entry n = k L + lane, so the lanes read
// neighbouring words), the sum over n ends with log2(L) shuffles. The request's tokens are walked in chunks of 8 with the next
// chunks on their way while this one is worked on: the B and C rows of three chunks by asynchronous copies into a ring of
// stages in shared memory, x, step sizes and gates of the next chunk as loads into registers that nothing reads before the
// chunk's turn. What a token needs once (its loads, the softplus, the gate, the store) is done by one lane of the channel for
// it, the lanes taking a chunk's tokens in turn, so it costs a chunk one pass and not eight; the walk gets a token's step size
// from its lane by a shuffle. The chain itself is one multiply-add per token and entry. Where the output is bfloat16 they use
// the special-function unit's exponential and logarithm. L and NS follow from `states` alone, so a row's operations do not
// depend on the step as long as its form does not; between the forms rows and state differ at rounding level.
#include "common.cuh"

namespace {

constexpr int SS_THREADS = 32;
constexpr int SS_CHUNK = 8;
constexpr int SS_AHEAD = 3;                // chunks whose inputs are under way beside the one at work
constexpr int SS_STAGES = SS_AHEAD + 1;

struct ScanArgs {
    const float* x; long x_t;
    const float* dt; long dt_t;
    const float* dt_bias;                 // [inner]
    const float* B; const float* C; long bc_t;
    const float* A;                       // [inner, states]
    const float* D;                       // [inner]
    const float* z; long z_t;             // or null
    float* state; long state_slot; long state_half;
    const int* q_start; const int* slots; const int* positions;
    void* out; long out_t;
    int inner, states, L;
};

// the recurrence's arithmetic in the accumulator's type: exact library functions for float64 (the true 32-bit path), the
// special-function unit for float32 (the bfloat16 path, whose products carry 8 bits)
__device__ __forceinline__ double ss_exp(double v) { return exp(v); }
__device__ __forceinline__ float ss_exp(float v) { return __expf(v); }
__device__ __forceinline__ double ss_softplus(double v) { return v > 20.0 ? v : log1p(exp(v)); }
__device__ __forceinline__ float ss_softplus(float v) { return v > 15.f ? v : __logf(1.f + __expf(v)); }

__device__ __forceinline__ void ss_cp_async_4(float* smem_dst, const float* gmem_src) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(gmem_src) : "memory");
}

template <typename T, typename ACC, int L, int NS>
__global__ void __launch_bounds__(SS_THREADS) selective_scan_kernel(const ScanArgs a) {
    extern __shared__ float bc_s[];                            // the ring: SS_STAGES stages of a chunk's inputs
    pdl_wait();                                    // what the kernels before wrote is complete
    pdl_trigger();
    constexpr int OWN = (SS_CHUNK + L - 1) / L;                // tokens of a chunk that a lane looks after
    const int r = blockIdx.x;
    const int Nst = a.states;
    constexpr int per_block = SS_THREADS / L;
    const int c = blockIdx.y * per_block + threadIdx.x / L;
    const int l = threadIdx.x % L;
    const bool ok = c < a.inner;
    const int begin = a.q_start[r], end = a.q_start[r + 1];
    if (end <= begin) return;
    const int p0 = a.positions[begin];
    float* slot = a.state + (size_t)a.slots[r] * a.state_slot;
    const float* rd = slot + ((p0 + 1) & 1) * a.state_half;
    float* wr = slot + ((p0 + end - begin - 1) & 1) * a.state_half;
    ACC S[NS];
    float A[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const int n = k * L + l;
        const bool have = ok && n < Nst;
        S[k] = have ? (ACC)rd[(size_t)c * Nst + n] : (ACC)0;
        A[k] = have ? a.A[(size_t)c * Nst + n] : 0.f;
    }
    const float dt_b = ok ? a.dt_bias[c] : 0.f;
    const float Dc = ok ? a.D[c] : 0.f;
    const bool gated = a.z != nullptr;
    T* out = reinterpret_cast<T*>(a.out);
    constexpr int CPW = SS_THREADS / L;                        // channels of the block
    const int stage_floats = SS_CHUNK * 2 * Nst;               // a chunk's rows [B | C]

    // a chunk's B and C rows go to a stage of the ring by 4-byte asynchronous copies, SS_AHEAD chunks before their turn
    auto copy_stage = [&](int t0, int nt, float* dst) {
        for (int tt = 0; tt < nt; ++tt) {
            for (int j = threadIdx.x; j < 2 * Nst; j += SS_THREADS)
                ss_cp_async_4(dst + tt * 2 * Nst + j, j < Nst ? a.B + (size_t)(t0 + tt) * a.bc_t + j : a.C + (size_t)(t0 + tt) * a.bc_t + j - Nst);
        }
        // rows past the portion's end take part in the chunk's arithmetic with step size 0: they must hold numbers
        for (int j = nt * 2 * Nst + threadIdx.x; j < SS_CHUNK * 2 * Nst; j += SS_THREADS) dst[j] = 0.f;
    };
    // a lane looks after the tokens l, l + L, .. of a chunk: it loads their x, step size and gate (a chunk ahead, into
    // registers that nothing reads before the chunk's turn), takes the softplus, and at the chunk's end gates and stores
    // their outputs; the walk gets a token's step size from its lane by a shuffle
    float xr[OWN], dr[OWN], zr[OWN];
    auto load_rows = [&](int t0, int nt, float (&xv)[OWN], float (&dv)[OWN], float (&zv)[OWN]) {
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
            const int tt = o * L + l;
            const bool have = ok && tt < nt;
            xv[o] = have ? a.x[(size_t)(t0 + tt) * a.x_t + c] : 0.f;
            dv[o] = have ? a.dt[(size_t)(t0 + tt) * a.dt_t + c] : 0.f;
            zv[o] = have && gated ? a.z[(size_t)(t0 + tt) * a.z_t + c] : 0.f;
        }
    };
    load_rows(begin, min(SS_CHUNK, end - begin), xr, dr, zr);
    const int chunks = (end - begin + SS_CHUNK - 1) / SS_CHUNK;
#pragma unroll
    for (int i = 0; i < SS_AHEAD; ++i) {
        if (i < chunks) copy_stage(begin + i * SS_CHUNK, min(SS_CHUNK, end - begin - i * SS_CHUNK), bc_s + i * stage_floats);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int i = 0; i < chunks; ++i) {
        const int t0 = begin + i * SS_CHUNK;
        const int nt = min(SS_CHUNK, end - t0);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(SS_AHEAD - 1) : "memory");
        __syncthreads();                                       // this chunk's stage is in; the stage read a round ago is free
        if (i + SS_AHEAD < chunks) {
            const int t1 = t0 + SS_AHEAD * SS_CHUNK;
            copy_stage(t1, min(SS_CHUNK, end - t1), bc_s + ((i + SS_AHEAD) % SS_STAGES) * stage_floats);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* rows = bc_s + (i % SS_STAGES) * stage_floats;
        float xn[OWN], dn[OWN], zn[OWN];
        const bool more = i + 1 < chunks;
        if (more) load_rows(t0 + SS_CHUNK, min(SS_CHUNK, end - t0 - SS_CHUNK), xn, dn, zn);
        // straight-line code for the chunk, so that the tokens' independent parts (shuffles, decays, the sums over the
        // lanes) overlap and only the multiply-adds on S form a chain. A token past the portion's end has step size 0:
        // decay 1 and nothing added.
        ACC dts[OWN], dxs[OWN], ys[OWN];
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
            dts[o] = o * L + l < nt ? ss_softplus((ACC)(dr[o] + dt_b)) : (ACC)0;
            dxs[o] = dts[o] * (ACC)xr[o];
            ys[o] = 0;
        }
        ACC dtv[SS_CHUNK], dxv[SS_CHUNK], yv[SS_CHUNK];
#pragma unroll
        for (int tt = 0; tt < SS_CHUNK; ++tt) {
            dtv[tt] = L > 1 ? __shfl_sync(0xffffffffu, dts[tt / L], tt % L, L) : dts[tt / L];
            dxv[tt] = L > 1 ? __shfl_sync(0xffffffffu, dxs[tt / L], tt % L, L) : dxs[tt / L];
            yv[tt] = 0;
        }
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const int n = k * L + l;
            const bool have = n < Nst;
            float Bv[SS_CHUNK], Cv[SS_CHUNK];
            ACC dA[SS_CHUNK];
#pragma unroll
            for (int tt = 0; tt < SS_CHUNK; ++tt) {
                Bv[tt] = have ? rows[tt * 2 * Nst + n] : 0.f;
                Cv[tt] = have ? rows[tt * 2 * Nst + Nst + n] : 0.f;
                dA[tt] = ss_exp(dtv[tt] * (ACC)A[k]);
            }
#pragma unroll
            for (int tt = 0; tt < SS_CHUNK; ++tt) {
                S[k] = fma(dA[tt], S[k], dxv[tt] * (ACC)Bv[tt]);
                yv[tt] = fma(S[k], (ACC)Cv[tt], yv[tt]);
            }
        }
#pragma unroll
        for (int w = L >> 1; w > 0; w >>= 1) {
#pragma unroll
            for (int tt = 0; tt < SS_CHUNK; ++tt) yv[tt] += __shfl_xor_sync(0xffffffffu, yv[tt], w);
        }
#pragma unroll
        for (int tt = 0; tt < SS_CHUNK; ++tt)
            if (tt % L == l) ys[tt / L] = yv[tt];
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
            const int tt = o * L + l;
            if (ok && tt < nt) {
                float yf = (float)fma((ACC)Dc, (ACC)xr[o], ys[o]);
                if (gated) yf *= sizeof(ACC) == 8 ? zr[o] / (1.f + expf(-zr[o])) : __fdividef(zr[o], 1.f + __expf(-zr[o]));
                out[(size_t)(t0 + tt) * a.out_t + c] = from_float<T>(yf);
            }
        }
        if (more) {
#pragma unroll
            for (int o = 0; o < OWN; ++o) { xr[o] = xn[o]; dr[o] = dn[o]; zr[o] = zn[o]; }
        }
    }
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const int n = k * L + l;
        if (ok && n < Nst) wr[(size_t)c * Nst + n] = (float)S[k];
    }
}

template <int L, int NS>
void launch_scan(const ScanArgs& a, int out_dtype, int R, cudaStream_t stream) {
    constexpr int per_block = SS_THREADS / L;
    dim3 grid(R, (unsigned)((a.inner + per_block - 1) / per_block));
    const size_t smem = (size_t)SS_STAGES * SS_CHUNK * 2 * a.states * sizeof(float);
    if (out_dtype == LLMP_BF16) {
        LLMP_ALLOW_SMEM((selective_scan_kernel<bf16, float, L, NS>), smem);
        llmp_launch_dependent(selective_scan_kernel<bf16, float, L, NS>, grid, dim3(SS_THREADS), smem, stream, a);
    } else {
        LLMP_ALLOW_SMEM((selective_scan_kernel<float, double, L, NS>), smem);
        llmp_launch_dependent(selective_scan_kernel<float, double, L, NS>, grid, dim3(SS_THREADS), smem, stream, a);
    }
}

// ---- many tokens: segments side by side --------------------------------------------------------------------------------
// The recurrence is linear in S, and over a run of tokens every entry decays by exp(A times the sum of the step sizes). So a
// request's tokens are cut into segments of SEG_TOKENS, counted from the portion's first token, and three launches take them:
//   1. every segment but a request's last, from a zero state: its own sum and the sum of its step sizes, to scratch;
//   2. along a request's segments: scratch becomes the state before each (requests of one segment have nothing to do);
//   3. every segment from the state before it: the outputs; the last segment leaves the state in the slot.
// Token by token, a prompt was one chain of 2,048 steps with 110 instructions a token and warp of two channels, most of them
// spent on what 16 lanes share. Here a thread holds a whole channel, so a token's step size, gate and sum over the entries
// cost once and the entries' multiply-adds go two at a time; the bound is then the special-function unit (an exponential per
// token and entry, in 1 and in 3: busy for 72 and 59 % of these launches). 2,048 tokens of 4,096 channels with 16 entries: 641 us
// token by token, 126 so (51, 18 and 68 with cold caches). Tried: three pairs of eight exponentials as polynomials on the
// multiply-add pipe (137 us), segments of 96 tokens (128), loads two tokens ahead (133), seven blocks an SM (126).
constexpr int SEG_TOKENS = 64;
constexpr int SEG_CHANNELS = 128;         // threads of a block, a channel each
constexpr int SEG_AHEAD = 4;              // tokens whose loads are under way while as many are worked on

struct SegArgs {
    ScanArgs s;
    float* sums;                          // [entries][inner][NS]: a segment's own sum, then the state before it
    float* steps;                         // [entries][inner]: sum of a segment's step sizes
    int requests;
};

struct Segment { int request, index, count, entry, begin, end; };

// Segment number `at` of the step (in the order of the requests); request -1: there is none. `entry`: its place in scratch,
// where requests of one segment have none. By a warp, every lane gets the answer.
__device__ __forceinline__ Segment find_segment(const int* q_start, int requests, int at) {
    const int lane = threadIdx.x & 31;
    int before = 0, entries = 0;
    Segment g;
    g.request = -1;
    for (int base = 0; base < requests; base += 32) {
        const int r = base + lane;
        const int first = r < requests ? q_start[r] : 0, last = r < requests ? q_start[r + 1] : 0;
        const int own = (max(last - first, 0) + SEG_TOKENS - 1) / SEG_TOKENS;
        int upto = own, kept = own > 1 ? own : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, upto, o), k = __shfl_up_sync(0xffffffffu, kept, o);
            if (lane >= o) { upto += u; kept += k; }
        }
        const unsigned reach = __ballot_sync(0xffffffffu, before + upto > at);
        if (reach) {
            const int src = __ffs(reach) - 1;
            g.request = base + src;
            g.count = __shfl_sync(0xffffffffu, own, src);
            g.index = at - before - (__shfl_sync(0xffffffffu, upto, src) - g.count);
            g.entry = entries + __shfl_sync(0xffffffffu, kept, src) - (g.count > 1 ? g.count : 0) + g.index;
            const int f = __shfl_sync(0xffffffffu, first, src), l = __shfl_sync(0xffffffffu, last, src);
            g.begin = f + g.index * SEG_TOKENS;
            g.end = min(l, g.begin + SEG_TOKENS);
            return g;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
        entries += __shfl_sync(0xffffffffu, kept, 31);
    }
    return g;
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)), "l"(reinterpret_cast<unsigned long long&>(c)));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return d;
}
__device__ __forceinline__ float ex2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
constexpr float LOG2_E = 1.4426950408889634f;

// OUT false: launch 1; true: launch 3. NS: state entries a thread holds, `states` rounded up (the others decay by 1 and stay 0).
template <int NS, bool OUT>
__global__ void __launch_bounds__(SEG_CHANNELS) scan_segments_kernel(const SegArgs g) {
    constexpr int W = OUT ? 2 * NS : NS;                       // entries of a token's row in shared memory: [B | C]
    __shared__ __align__(16) float bc[SEG_TOKENS * W];
    pdl_wait();
    pdl_trigger();
    const ScanArgs& a = g.s;
    const Segment seg = find_segment(a.q_start, g.requests, blockIdx.x);
    if (seg.request < 0 || (!OUT && seg.index + 1 == seg.count)) return;
    const int cnt = seg.end - seg.begin, states = a.states;
    for (int i = threadIdx.x; i < cnt * W; i += SEG_CHANNELS) {
        const int t = i / W, j = i % W, n = j % NS;
        const float* row = (j < NS ? a.B : a.C) + (size_t)(seg.begin + t) * a.bc_t;
        bc[i] = n < states ? row[n] : 0.f;
    }
    const int c = blockIdx.y * SEG_CHANNELS + threadIdx.x;
    const bool ok = c < a.inner;
    float2 S[NS / 2], A[NS / 2];
    const int p0 = a.positions[seg.begin - seg.index * SEG_TOKENS];
    float* slot = a.state + (size_t)a.slots[seg.request] * a.state_slot + (size_t)c * states;
    {
        float from[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) from[n] = 0.f;
        if (OUT && ok) {
            if (seg.count > 1) {
                const float4* at = reinterpret_cast<const float4*>(g.sums + ((size_t)seg.entry * a.inner + c) * NS);
#pragma unroll
                for (int n = 0; n < NS / 4; ++n) {
                    const float4 v = at[n];
                    from[4 * n] = v.x; from[4 * n + 1] = v.y; from[4 * n + 2] = v.z; from[4 * n + 3] = v.w;
                }
            } else {
                const float* rd = slot + ((p0 + 1) & 1) * a.state_half;
#pragma unroll
                for (int n = 0; n < NS; ++n)
                    if (n < states) from[n] = rd[n];
            }
        }
#pragma unroll
        for (int n = 0; n < NS; n += 2) {
            S[n / 2] = make_float2(from[n], from[n + 1]);
            A[n / 2].x = ok && n < states ? a.A[(size_t)c * states + n] * LOG2_E : 0.f;
            A[n / 2].y = ok && n + 1 < states ? a.A[(size_t)c * states + n + 1] * LOG2_E : 0.f;
        }
    }
    const float dt_b = ok ? a.dt_bias[c] : 0.f;
    const float Dc = OUT && ok ? a.D[c] : 0.f;
    const bool gated = OUT && a.z != nullptr;
    const int cc = ok ? c : 0;
    const float* xp = a.x + (size_t)seg.begin * a.x_t + cc;
    const float* dp = a.dt + (size_t)seg.begin * a.dt_t + cc;
    const float* zp = gated ? a.z + (size_t)seg.begin * a.z_t + cc : xp;
    bf16* out = reinterpret_cast<bf16*>(a.out) + (size_t)seg.begin * a.out_t + cc;
    const int x_t = (int)a.x_t, d_t = (int)a.dt_t, z_t = gated ? (int)a.z_t : x_t, o_t = (int)a.out_t;
    float xn[SEG_AHEAD], dn[SEG_AHEAD], zn[SEG_AHEAD];
    auto load = [&](int t0) {                                  // past the end: the last token's again, which nothing uses
#pragma unroll
        for (int u = 0; u < SEG_AHEAD; ++u) {
            const int t = min(t0 + u, cnt - 1);
            xn[u] = xp[t * x_t];
            dn[u] = dp[t * d_t];
            if (OUT) zn[u] = zp[t * z_t];
        }
    };
    float walked = 0.f;
    auto step = [&](int t, float x, float raw, float z) {
        const float dt = ss_softplus(raw + dt_b);
        const float2 dt2 = make_float2(dt, dt), dx2 = make_float2(dt * x, dt * x);
        const float4* row = reinterpret_cast<const float4*>(bc + t * W);
        float2 y2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int n = 0; n < NS / 4; ++n) {
            const float4 b = row[n];
            const float2 e0 = mul2(dt2, A[2 * n]), e1 = mul2(dt2, A[2 * n + 1]);
            S[2 * n] = fma2(make_float2(ex2(e0.x), ex2(e0.y)), S[2 * n], mul2(dx2, make_float2(b.x, b.y)));
            S[2 * n + 1] = fma2(make_float2(ex2(e1.x), ex2(e1.y)), S[2 * n + 1], mul2(dx2, make_float2(b.z, b.w)));
            if (OUT) {
                const float4 r = row[NS / 4 + n];
                y2 = fma2(S[2 * n], make_float2(r.x, r.y), y2);
                y2 = fma2(S[2 * n + 1], make_float2(r.z, r.w), y2);
            }
        }
        if (OUT) {
            float y = fmaf(Dc, x, y2.x + y2.y);
            if (gated) y *= __fdividef(z, 1.f + __expf(-z));
            if (ok) out[t * o_t] = __float2bfloat16_rn(y);
        } else {
            walked += dt;
        }
    };
    load(0);
    __syncthreads();
    int t0 = 0;
    for (; t0 + SEG_AHEAD <= cnt; t0 += SEG_AHEAD) {
        float xv[SEG_AHEAD], dv[SEG_AHEAD], zv[SEG_AHEAD];
#pragma unroll
        for (int u = 0; u < SEG_AHEAD; ++u) { xv[u] = xn[u]; dv[u] = dn[u]; zv[u] = OUT ? zn[u] : 0.f; }
        load(t0 + SEG_AHEAD);
#pragma unroll
        for (int u = 0; u < SEG_AHEAD; ++u) step(t0 + u, xv[u], dv[u], zv[u]);
    }
#pragma unroll
    for (int u = 0; u < SEG_AHEAD - 1; ++u)
        if (t0 + u < cnt) step(t0 + u, xn[u], dn[u], OUT ? zn[u] : 0.f);
    if (!ok) return;
    if (!OUT) {
        float4* to = reinterpret_cast<float4*>(g.sums + ((size_t)seg.entry * a.inner + c) * NS);
#pragma unroll
        for (int n = 0; n < NS / 4; ++n) to[n] = make_float4(S[2 * n].x, S[2 * n].y, S[2 * n + 1].x, S[2 * n + 1].y);
        g.steps[(size_t)seg.entry * a.inner + c] = walked;
    } else if (seg.index + 1 == seg.count) {
        const int tokens = seg.end - seg.begin + seg.index * SEG_TOKENS;
        float* wr = slot + ((p0 + tokens - 1) & 1) * a.state_half;
#pragma unroll
        for (int n = 0; n < NS; n += 2) {
            if (n < states) wr[n] = S[n / 2].x;
            if (n + 1 < states) wr[n + 1] = S[n / 2].y;
        }
    }
}

// Launch 2: a thread per state entry of a request walks its segments. It reads the slot here and not in launch 3, whose last
// segment may write the very copy that the first would read.
template <int NS>
__global__ void __launch_bounds__(256) scan_states_kernel(const SegArgs g) {
    pdl_wait();
    pdl_trigger();
    const ScanArgs& a = g.s;
    const int r = blockIdx.y, lane = threadIdx.x & 31;
    const int begin = a.q_start[r], tokens = a.q_start[r + 1] - begin;
    const int count = (max(tokens, 0) + SEG_TOKENS - 1) / SEG_TOKENS;
    if (count <= 1) return;
    int before = 0;                                            // entries of the requests in front
    for (int i = lane; i < r; i += 32) {
        const int own = (max(a.q_start[i + 1] - a.q_start[i], 0) + SEG_TOKENS - 1) / SEG_TOKENS;
        if (own > 1) before += own;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    const int i = blockIdx.x * 256 + threadIdx.x, c = i / NS, n = i % NS;
    if (c >= a.inner) return;
    const float A = n < a.states ? a.A[(size_t)c * a.states + n] * LOG2_E : 0.f;
    float S = 0.f;
    if (n < a.states) S = a.state[(size_t)a.slots[r] * a.state_slot + ((a.positions[begin] + 1) & 1) * a.state_half + (size_t)c * a.states + n];
    float* at = g.sums + ((size_t)before * a.inner + c) * NS + n;
    const float* step = g.steps + (size_t)before * a.inner + c;
    const size_t stride = (size_t)a.inner * NS;
    constexpr int AHEAD = 8;
    float own[AHEAD], dt[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
        own[k] = k + 1 < count ? at[k * stride] : 0.f;
        dt[k] = k + 1 < count ? step[(size_t)k * a.inner] : 0.f;
    }
    for (int s = 0; s < count; s += AHEAD) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if (s + k >= count) break;
            const float u = own[k], d = dt[k];
            const int next = s + k + AHEAD;
            if (next + 1 < count) { own[k] = at[next * stride]; dt[k] = step[(size_t)next * a.inner]; }
            at[(s + k) * stride] = S;
            S = fmaf(ex2(A * d), S, u);
        }
    }
}

template <int NS>
void launch_segments(const SegArgs& g, int segments, cudaStream_t stream) {
    const dim3 grid(segments, (unsigned)((g.s.inner + SEG_CHANNELS - 1) / SEG_CHANNELS));
    if (g.sums) {                                              // null: no request has two segments
        llmp_launch_dependent(scan_segments_kernel<NS, false>, grid, dim3(SEG_CHANNELS), 0, stream, g);
        const dim3 states((unsigned)(((long)g.s.inner * NS + 255) / 256), g.requests);
        llmp_launch_dependent(scan_states_kernel<NS>, states, dim3(256), 0, stream, g);
    }
    llmp_launch_dependent(scan_segments_kernel<NS, true>, grid, dim3(SEG_CHANNELS), 0, stream, g);
}

}  // namespace

LLMP_API int llmp_selective_scan_segments(const float* x, long x_t, const float* dt, long dt_t, const float* dt_bias, const float* B,
                                          const float* C, long bc_t, const float* A, const float* D, const float* z, long z_t, float* state,
                                          long state_slot, long state_half, const int* q_start, const int* slots, const int* positions,
                                          void* out, long out_t, float* scratch, long scratch_floats, int rows, int R, int inner,
                                          int states, cudaStream_t stream) {
    if (R <= 0 || rows <= 0) return 0;
    const int padded = states <= 8 ? 8 : states <= 16 ? 16 : 32;
    for (long stride : {x_t, dt_t, z_t, out_t})                // offsets within a segment are 32-bit
        LLMP_REQUIRE(stride >= 0 && stride < (1l << 24), "selective_scan: a row stride of %ld entries", stride);
    LLMP_REQUIRE(inner > 0 && states > 0 && states <= padded, "selective_scan: %d channels with %d state entries (segments: up to 32 entries)", inner, states);
    LLMP_REQUIRE(state_half >= (long)inner * states, "selective_scan: the state piece is shorter than the state");
    LLMP_REQUIRE(R <= 65535 && (inner + SEG_CHANNELS - 1) / SEG_CHANNELS <= 65535, "selective_scan: too many channels %d or requests %d", inner, R);
    const int more = (rows - 1) / SEG_TOKENS;                  // segments beyond the first of each request, at most
    const long entries = more + (more < R ? more : R);
    LLMP_REQUIRE(scratch_floats >= entries * inner * (padded + 1) && (entries == 0 || scratch), "selective_scan: segments need %ld floats of scratch",
                 entries * inner * (padded + 1));
    SegArgs g;
    ScanArgs& a = g.s;
    a.x = x; a.x_t = x_t; a.dt = dt; a.dt_t = dt_t; a.dt_bias = dt_bias; a.B = B; a.C = C; a.bc_t = bc_t; a.A = A; a.D = D;
    a.z = z; a.z_t = z_t; a.state = state; a.state_slot = state_slot; a.state_half = state_half; a.q_start = q_start;
    a.slots = slots; a.positions = positions; a.out = out; a.out_t = out_t; a.inner = inner; a.states = states; a.L = 0;
    g.sums = entries ? scratch : nullptr; g.steps = scratch + entries * inner * padded; g.requests = R;
    const int segments = more + R;
    if (padded == 8) launch_segments<8>(g, segments, stream);
    else if (padded == 16) launch_segments<16>(g, segments, stream);
    else launch_segments<32>(g, segments, stream);
    return llmp_check_launch("selective_scan_segments");
}

LLMP_API int llmp_selective_scan(const float* x, long x_t, const float* dt, long dt_t, const float* dt_bias, const float* B,
                                 const float* C, long bc_t, const float* A, const float* D, const float* z, long z_t, float* state,
                                 long state_slot, long state_half, const int* q_start, const int* slots, const int* positions,
                                 void* out, int out_dtype, long out_t, int R, int inner, int states, cudaStream_t stream) {
    if (R <= 0) return 0;
    LLMP_REQUIRE(inner > 0 && states > 0 && states <= 256, "selective_scan: %d channels with %d state entries (up to 256 are served)",
                 inner, states);
    LLMP_REQUIRE(state_half >= (long)inner * states, "selective_scan: the state piece is shorter than the state");
    // a lane per state entry up to 32 entries, then 32 lanes with more each: a long prompt is a chain of dependent steps
    // per warp, and what hides their latency is the number of warps (measured: 0.59 ms for 2,048 tokens of 4,096 channels
    // with 16 entries so; 1.08 ms with 8 entries a lane, a sixth of the instructions but an eighth of the warps)
    int L = 1;
    while (L < 32 && L < states) L *= 2;
    const int NS = (states + L - 1) / L;
    ScanArgs a;
    a.x = x; a.x_t = x_t; a.dt = dt; a.dt_t = dt_t; a.dt_bias = dt_bias; a.B = B; a.C = C; a.bc_t = bc_t; a.A = A; a.D = D;
    a.z = z; a.z_t = z_t; a.state = state; a.state_slot = state_slot; a.state_half = state_half; a.q_start = q_start;
    a.slots = slots; a.positions = positions; a.out = out; a.out_t = out_t; a.inner = inner; a.states = states; a.L = L;
    LLMP_REQUIRE(((long)inner * L + SS_THREADS - 1) / SS_THREADS <= 65535, "selective_scan: too many channels %d", inner);
    switch (L) {
        case 1: launch_scan<1, 1>(a, out_dtype, R, stream); break;
        case 2: launch_scan<2, 1>(a, out_dtype, R, stream); break;
        case 4: launch_scan<4, 1>(a, out_dtype, R, stream); break;
        case 8: launch_scan<8, 1>(a, out_dtype, R, stream); break;
        case 16: launch_scan<16, 1>(a, out_dtype, R, stream); break;
        default:
            if (NS <= 1) launch_scan<32, 1>(a, out_dtype, R, stream);
            else if (NS <= 2) launch_scan<32, 2>(a, out_dtype, R, stream);
            else if (NS <= 4) launch_scan<32, 4>(a, out_dtype, R, stream);
            else launch_scan<32, 8>(a, out_dtype, R, stream);
    }
    return llmp_check_launch("selective_scan");
}
