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
// G lanes share a channel and hold E neighbouring state entries each; the lanes' sums are added in one fixed order. G and E follow
// from `states` alone and the first two forms do the same operations in the same order, so a row and the state after it have the same
// bits in any company.
//   step: requests of a single token. A thread loads its entries, takes the step and stores them: the state is read and written once
//         (8 requests of 4,096 channels with 16 entries 3.5 us; 17.9 as a walk).
//   walk: a block takes a request and the channels of its walking warps, token by token. A walk needs each exponential once (segments
//         twice), so the special-function unit would be done with 2,048 tokens of 4,096 channels in 37 us; what keeps a walk from that
//         is that a scheduler has one or two warps of it, which wait for every instruction's result. So whatever the chain does not
//         need is other warps' work (copies into a ring, step sizes and gates of the stages to come, the sums over a channel's lanes and
//         the outputs of the stage behind; they meet the walkers at one barrier a stage), and a walker's turn of up to four tokens mixes
//         three: the chain over one run, the decays of the next, the loads of the one after. Microseconds, before and after: 2,048
//         tokens of 4,096 channels 117 (segments) and 94, of 2,048 channels 84 and 54; 100 tokens 33 and 9; 203 in float64 68 and 31;
//         64 single tokens beside 300 102 and 57; with 64, 128 and 256 entries, 1,024 tokens of 2,048 channels 728, 1,772 and 5,478 and
//         189, 310 and 623. On the way: all of it in one warp 209 and 149, sums by shuffles among the walkers 155
//         and 106, stages of 16 tokens 109 and 84, two warps for step sizes and gates 104 and 74.
//   segments: few channels and many tokens in bfloat16 (below).
#include <type_traits>

#include "common.cuh"

namespace {

// Tokens of a turn of the walk, by the entries a lane holds: a turn's two sets of registers are twelve a token and entry in float64,
// eight in float32. Four tokens of four or eight entries spilled up to 3,816 bytes a thread.
template <typename ACC, int E> constexpr int SS_RUN = (int)sizeof(ACC) * E <= 16 ? 4 : (int)sizeof(ACC) * E <= 32 ? 2 : 1;
// threads of a block that walk; then come a warp that copies, four for step sizes and gates, two for the outputs
template <int G> constexpr int SS_WALKERS = G < 8 ? 64 : 128;

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
    int inner, states, requests;
    int held;                             // 1: no kernel in flight writes A, D or dt_bias
    int singles;                          // 1: the walk leaves requests of one token to the step kernel
};

// The arithmetic in the accumulator's type: exact library functions for float64 (the true 32-bit path), the special-function
// unit for float32 (the bfloat16 path, whose products carry 8 bits). Decays: 2 to the power of the step size times A log2(e) there.
__device__ __forceinline__ double ss_softplus(double v) { return v > 20.0 ? v : log1p(exp(v)); }
__device__ __forceinline__ float ss_softplus(float v) { return v > 15.f ? v : __logf(1.f + __expf(v)); }
__device__ __forceinline__ float ss_gate(float z, double) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float ss_gate(float z, float) { return __fdividef(z, 1.f + __expf(-z)); }
constexpr float LOG2_E = 1.4426950408889634f;
__device__ __forceinline__ double ss_rate(float a, double) { return (double)a; }
__device__ __forceinline__ float ss_rate(float a, float) { return a * LOG2_E; }

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

// A token's decays of a lane's E entries and what it adds to them; then S <- decay S + add, and the lane's share of sum S C.
template <int E>
__device__ __forceinline__ void ss_decays(const float (&A)[E], float dt, float dx, const float* b, float (&decay)[E], float (&add)[E]) {
    const float2 dt2 = make_float2(dt, dt), dx2 = make_float2(dx, dx);
#pragma unroll
    for (int e = 0; e < E; e += 2) {
        const float2 p = mul2(dt2, make_float2(A[e], A[e + 1])), q = mul2(dx2, make_float2(b[e], b[e + 1]));
        decay[e] = ex2(p.x); decay[e + 1] = ex2(p.y);
        add[e] = q.x; add[e + 1] = q.y;
    }
}
template <int E>
__device__ __forceinline__ float ss_advance(float (&S)[E], const float (&decay)[E], const float (&add)[E], const float* c) {
    float2 y = make_float2(0.f, 0.f);
#pragma unroll
    for (int e = 0; e < E; e += 2) {
        const float2 s = fma2(make_float2(decay[e], decay[e + 1]), make_float2(S[e], S[e + 1]), make_float2(add[e], add[e + 1]));
        S[e] = s.x; S[e + 1] = s.y;
        y = e ? fma2(s, make_float2(c[e], c[e + 1]), y) : mul2(s, make_float2(c[e], c[e + 1]));
    }
    return y.x + y.y;
}
template <int E>
__device__ __forceinline__ void ss_decays(const double (&A)[E], double dt, double dx, const float* b, double (&decay)[E], double (&add)[E]) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
        decay[e] = exp(dt * A[e]);
        add[e] = dx * (double)b[e];
    }
}
template <int E>
__device__ __forceinline__ double ss_advance(double (&S)[E], const double (&decay)[E], const double (&add)[E], const float* c) {
    double y = 0.0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        S[e] = fma(decay[e], S[e], add[e]);
        y = fma(S[e], (double)c[e], y);
    }
    return y;
}
__device__ __forceinline__ void ss_pair(const unsigned char* p, float (&d)[2]) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    d[0] = v.x; d[1] = v.y;
}
__device__ __forceinline__ void ss_pair(const unsigned char* p, double (&d)[2]) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    d[0] = v.x; d[1] = v.y;
}

__device__ __forceinline__ void ss_put2(unsigned char* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void ss_put2(unsigned char* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }
// A lane's sums of a run's tokens, and the sums of them over the G lanes of a channel, in the order of ss_reduce.
template <int RUN, typename ACC> __device__ __forceinline__ void ss_put(unsigned char* p, const ACC (&v)[RUN]) {
    if constexpr (RUN == 1) *reinterpret_cast<ACC*>(p) = v[0];
    else if constexpr (RUN == 4 && sizeof(ACC) == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else {
#pragma unroll
        for (int t = 0; t < RUN; t += 2) ss_put2(p + t * sizeof(ACC), v[t], v[t + 1]);
    }
}
template <int RUN, typename ACC> __device__ __forceinline__ void ss_get(const unsigned char* p, ACC (&v)[RUN]) {
    if constexpr (RUN == 1) v[0] = *reinterpret_cast<const ACC*>(p);
    else if constexpr (RUN == 4 && sizeof(ACC) == 4) {
        const float4 u = *reinterpret_cast<const float4*>(p);
        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
    } else {
#pragma unroll
        for (int t = 0; t < RUN; t += 2) {
            ACC u[2];
            ss_pair(p + t * sizeof(ACC), u);
            v[t] = u[0]; v[t + 1] = u[1];
        }
    }
}
template <int G, int RUN, typename ACC> __device__ __forceinline__ void ss_gather(const unsigned char* p, ACC (&y)[RUN]) {
    constexpr int PITCH = RUN * sizeof(ACC);
    ACC v[G / 2][RUN];
#pragma unroll
    for (int i = 0; i < G / 2; ++i) {
        ACC u[RUN];
        ss_get(p + i * PITCH, v[i]);
        ss_get(p + (i + G / 2) * PITCH, u);
#pragma unroll
        for (int t = 0; t < RUN; ++t) v[i][t] += u[t];
    }
#pragma unroll
    for (int w = G / 4; w > 0; w >>= 1)
#pragma unroll
        for (int i = 0; i < w; ++i)
#pragma unroll
            for (int t = 0; t < RUN; ++t) v[i][t] += v[i + w][t];
#pragma unroll
    for (int t = 0; t < RUN; ++t) y[t] = v[0][t];
}
template <int G, typename ACC> __device__ __forceinline__ ACC ss_reduce(ACC y) {
#pragma unroll
    for (int w = G >> 1; w > 0; w >>= 1) y += __shfl_xor_sync(0xffffffffu, y, w);
    return y;
}

// Entry e of a lane's E neighbours at `p`; `have` of them exist, the others read 0.
template <int E, typename ACC>
__device__ __forceinline__ void ss_load(ACC (&v)[E], const float* p, int have) {
    if (have >= E && (uintptr_t)p % (E < 4 ? 8 : 16) == 0) {
        if (E == 2) {
            const float2 u = *reinterpret_cast<const float2*>(p);
            v[0] = u.x; v[1] = u.y;
        } else {
#pragma unroll
            for (int e = 0; e < E; e += 4) {
                const float4 u = *reinterpret_cast<const float4*>(p + e);
                v[e] = u.x; v[(e + 1) % E] = u.y; v[(e + 2) % E] = u.z; v[(e + 3) % E] = u.w;
            }
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = e < have ? p[e] : 0.f;
}
template <int E, typename ACC>
__device__ __forceinline__ void ss_store(const ACC (&v)[E], float* p, int have) {
    if (have >= E && (uintptr_t)p % (E < 4 ? 8 : 16) == 0) {
        if (E == 2) {
            *reinterpret_cast<float2*>(p) = make_float2((float)v[0], (float)v[1]);
        } else {
#pragma unroll
            for (int e = 0; e < E; e += 4)
                *reinterpret_cast<float4*>(p + e) = make_float4((float)v[e], (float)v[(e + 1) % E], (float)v[(e + 2) % E], (float)v[(e + 3) % E]);
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (e < have) p[e] = (float)v[e];
}


// A request's single token.
template <typename T, typename ACC, int G, int E>
__global__ void __launch_bounds__(SS_WALKERS<G>) selective_step_kernel(const ScanArgs a) {
    constexpr int CH = SS_WALKERS<G> / G;
    const int r = blockIdx.x % a.requests, l = threadIdx.x % G;
    const int c = blockIdx.x / a.requests * CH + threadIdx.x / G;
    const bool ok = c < a.inner;
    const int cc = ok ? c : 0, have = ok ? a.states - l * E : 0;
    float rate[E], bias, Dc;
    auto load_layer = [&]() {
        ss_load<E>(rate, a.A + (size_t)cc * a.states + l * E, have);
        bias = a.dt_bias[cc];
        Dc = a.D[cc];
    };
    if (a.held) load_layer();                                   // (a decoding layer 34.6 us without, 32.9 so)
    pdl_wait();                                                 // what the kernels before wrote is complete
    pdl_trigger();
    if (!a.held) load_layer();
    const int t = a.q_start[r];
    if (a.q_start[r + 1] - t != 1) return;
    const int p0 = a.positions[t];
    float* slot = a.state + (size_t)a.slots[r] * a.state_slot + (size_t)cc * a.states + l * E;
    ACC S[E], A[E];
    ss_load<E>(S, slot + ((p0 + 1) & 1) * a.state_half, have);
    float b[E], k[E];
    ss_load<E>(b, a.B + (size_t)t * a.bc_t + l * E, a.states - l * E);
    ss_load<E>(k, a.C + (size_t)t * a.bc_t + l * E, a.states - l * E);
    const float x = a.x[(size_t)t * a.x_t + cc], raw = a.dt[(size_t)t * a.dt_t + cc];
    const float z = a.z ? a.z[(size_t)t * a.z_t + cc] : 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) A[e] = ss_rate(rate[e], ACC());
    const ACC dt = ss_softplus((ACC)(raw + bias));
    ACC decay[E], add[E];
    ss_decays<E>(A, dt, dt * (ACC)x, b, decay, add);
    const ACC y = ss_reduce<G>(ss_advance<E>(S, decay, add, k));
    ss_store<E>(S, slot + (p0 & 1) * a.state_half, have);
    if (ok && l == 0) {
        float o = (float)fma((ACC)Dc, (ACC)x, y);
        if (a.z) o *= ss_gate(z, ACC());
        reinterpret_cast<T*>(a.out)[(size_t)t * a.out_t + c] = from_float<T>(o);
    }
}

template <int BYTES>
__device__ __forceinline__ void ss_copy(float* dst, const float* src, bool have) {      // not there: zeros
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = have ? BYTES : 0;
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;\n" ::"r"(d), "l"(src), "r"(n), "n"(BYTES) : "memory");
}

// Shared memory of a walk: a ring of stages, each the x, dt and z rows of STAGE tokens [token][channel] and their B and C in the
// order of a channel's lanes ([token][lane][E of B | E of C]); three buffers of step sizes [channel][token] (step size, step size
// times x); two of the lanes' sums [run][channel][lane][RUN tokens]. The pitches spread a warp's channels over the banks.
template <typename ACC, int G, int E> struct ScanSmem {
    static constexpr int CH = SS_WALKERS<G> / G, P = G * E, RUN = SS_RUN<ACC, E>;
    static constexpr int STAGE = P > 64 || CH > 16 ? 16 : 32;  // tokens; two blocks an SM where that can be
    static constexpr int STAGES = 5;                           // one walked, one behind it, two before it, one under way
    static constexpr int ROWS = STAGE * CH;
    static constexpr int STAGE_FLOATS = 3 * ROWS + STAGE * 2 * P;
    static constexpr int STEP_PITCH = STAGE * 2 * (int)sizeof(ACC) + 16;          // bytes
    static constexpr int SUM_PITCH = G * RUN * (int)sizeof(ACC) + 16, SUM_BYTES = STAGE / RUN * CH * SUM_PITCH;
    static constexpr size_t BYTES = (size_t)STAGES * STAGE_FLOATS * 4 + 3 * CH * STEP_PITCH + 2 * SUM_BYTES;
    static_assert(BYTES <= 227 * 1024 && STAGE % (2 * RUN) == 0, "a block's shared memory; a stage is whole turns");
};

// WIDE: x, dt and z rows may be copied by 16 bytes (alignment, and `inner` a multiple of the block's channels), B and C by E floats, and
// rows lie less than 2^31 entries apart. The blocks are along x, which holds them for any number of channels and requests.
// Requests of a single token are left to the step kernel where `singles` says that it runs too.
template <typename T, typename ACC, int G, int E, bool WIDE>
__global__ void __launch_bounds__(SS_WALKERS<G> + 224, E == 2 && sizeof(ACC) == 4 ? 2 : 1) selective_walk_kernel(const ScanArgs a) {
    typedef ScanSmem<ACC, G, E> L;
    constexpr int CH = L::CH, P = L::P, STAGE = L::STAGE, RUN = L::RUN;
    extern __shared__ __align__(16) float ss_smem[];
    unsigned char* const steps = reinterpret_cast<unsigned char*>(ss_smem + L::STAGES * L::STAGE_FLOATS);
    unsigned char* const sums = steps + 3 * CH * L::STEP_PITCH;
    const int r = blockIdx.x % a.requests, tid = threadIdx.x, c0 = blockIdx.x / a.requests * CH;
    pdl_wait();                                                // what the kernels before wrote is complete
    pdl_trigger();
    const int begin = a.q_start[r], n = a.q_start[r + 1] - begin;
    if (n <= a.singles) return;
    const int stages = (n + STAGE - 1) / STAGE;

    if (tid < SS_WALKERS<G>) {
        const int l = tid % G, lc = tid / G, c = c0 + lc;      // lane of its channel, channel of the block
        const bool ok = c < a.inner;
        const int cc = ok ? c : 0, have = ok ? a.states - l * E : 0;
        const int p0 = a.positions[begin];
        float* slot = a.state + (size_t)a.slots[r] * a.state_slot + (size_t)cc * a.states + l * E;
        ACC S[E], A[E];
        {
            float rate[E];
            ss_load<E>(rate, a.A + (size_t)cc * a.states + l * E, have);
#pragma unroll
            for (int e = 0; e < E; ++e) A[e] = ss_rate(rate[e], ACC());
        }
        ss_load<E>(S, slot + ((p0 + 1) & 1) * a.state_half, have);
        // In turn j: decays of run j + 1, the chain over run j, the rows of run j + 2 from shared memory. Nothing in a turn waits for
        // another part of it. Two sets of registers take turns.
        ACC decay[2][RUN][E], add[2][RUN][E], step[2][RUN][2];
        float rows[2][RUN][2 * E];                          // B | C
        const float* const bc0 = ss_smem + 3 * L::ROWS + l * 2 * E;
        const unsigned char* const step0 = steps + lc * L::STEP_PITCH;
        unsigned char* const sum0 = sums + lc * L::SUM_PITCH + l * RUN * sizeof(ACC);
        constexpr int RUN_BC = RUN * 2 * P, RUN_STEP = RUN * 2 * (int)sizeof(ACC), RUN_SUM = CH * L::SUM_PITCH;
        auto fetch = [&](int set, const float* bc, const unsigned char* st) {
#pragma unroll
            for (int t = 0; t < RUN; ++t) {
                ss_pair(st + t * 2 * sizeof(ACC), step[set][t]);
                const float4* at = reinterpret_cast<const float4*>(bc + t * 2 * P);
#pragma unroll
                for (int i = 0; i < E / 2; ++i) {
                    const float4 w = at[i];
                    rows[set][t][4 * i] = w.x; rows[set][t][4 * i + 1] = w.y; rows[set][t][4 * i + 2] = w.z; rows[set][t][4 * i + 3] = w.w;
                }
            }
        };
        auto decays = [&](int set) {
#pragma unroll
            for (int t = 0; t < RUN; ++t) ss_decays<E>(A, step[set][t][0], step[set][t][1], rows[set][t], decay[set][t], add[set][t]);
        };
        __syncthreads();                                       // the first stages are in
        __syncthreads();                                       // and the first two's step sizes there
        fetch(0, bc0, step0);
        fetch(1, bc0 + RUN_BC, step0 + RUN_STEP);
        decays(0);
        int ring = 0, buffer = 0;                              // of this stage
        for (int s = 0; s < stages; ++s) {
            const int ring1 = ring + 1 == L::STAGES ? 0 : ring + 1, buffer1 = buffer == 2 ? 0 : buffer + 1;
            const float* bc = bc0 + ring * L::STAGE_FLOATS;
            const unsigned char* st = step0 + buffer * CH * L::STEP_PITCH;
            unsigned char* to = sum0 + (s & 1) * L::SUM_BYTES;
#pragma unroll 1
            for (int t0 = 0; t0 < min(STAGE, n - s * STAGE); t0 += 2 * RUN) {
                const bool last = t0 + 2 * RUN == STAGE;    // then the runs to fetch are the next stage's first two
                bc = last ? bc0 + ring1 * L::STAGE_FLOATS : bc + 2 * RUN_BC;
                st = last ? step0 + buffer1 * CH * L::STEP_PITCH : st + 2 * RUN_STEP;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    ACC part[RUN];
                    decays(u ^ 1);
#pragma unroll
                    for (int t = 0; t < RUN; ++t) part[t] = ss_advance<E>(S, decay[u][t], add[u][t], rows[u][t] + E);
                    fetch(u, bc + u * RUN_BC, st + u * RUN_STEP);
                    ss_put(to, part);
                    to += RUN_SUM;
                }
            }
            ring = ring1;
            buffer = buffer1;
            __syncthreads();
        }
        ss_store<E>(S, slot + ((p0 + n - 1) & 1) * a.state_half, have);
        return;
    }

    const bool gated = a.z != nullptr;
    if (tid < SS_WALKERS<G> + 32) {
        // Stage s of the ring <- its STAGE tokens; zeros past the end. A lane copies the same places of every stage: of the rows of x,
        // dt and z the floats at xq of every xt-th token, of the rows B | C likewise.
        const int h = tid % 32;
        constexpr int XU = WIDE ? 4 : 1, XCOLS = CH / XU, XT = 32 / XCOLS, BU = WIDE ? (E < 4 ? E : 4) : 1, BCOLS = 2 * P / BU;
        constexpr int BT = 32 >= BCOLS ? 32 / BCOLS : 1, BJ = BCOLS >= 32 ? BCOLS / 32 : 1;
        const int xq = h % XCOLS * XU, x0 = h / XCOLS, b0 = h / BCOLS;
        const bool in_x = c0 + xq < a.inner;
        const float* px = a.x + (size_t)begin * a.x_t + (in_x ? c0 + xq : 0);
        const float* pd = a.dt + (size_t)begin * a.dt_t + (in_x ? c0 + xq : 0);
        const float* pz = gated ? a.z + (size_t)begin * a.z_t + (in_x ? c0 + xq : 0) : a.x;
        typedef std::conditional_t<WIDE, int, long> Stride;
        const Stride x_t = (Stride)a.x_t, d_t = (Stride)a.dt_t, z_t = (Stride)a.z_t, bc_t = (Stride)a.bc_t;
        auto copy_stage = [&](int s) {
            if (s < stages) {
                float* st = ss_smem + (s % L::STAGES) * L::STAGE_FLOATS;
                const int t0 = s * STAGE, nt = n - t0;
                const float* sx = px + (size_t)t0 * a.x_t;
                const float* sd = pd + (size_t)t0 * a.dt_t;
                const float* sz = gated ? pz + (size_t)t0 * a.z_t : pz;
#pragma unroll
                for (int i = 0; i < (STAGE + XT - 1) / XT; ++i) {
                    const int t = x0 + i * XT;
                    if (XT > STAGE && t >= STAGE) break;
                    const bool in = t < nt && in_x;
                    const int row = in ? t : 0;
                    float* d = st + t * CH + xq;
                    ss_copy<XU * 4>(d, sx + (long)row * x_t, in);
                    ss_copy<XU * 4>(d + L::ROWS, sd + (long)row * d_t, in);
                    if (gated) ss_copy<XU * 4>(d + 2 * L::ROWS, sz + (long)row * z_t, in);
                }
#pragma unroll (WIDE && BJ == 2 ? 2 : 1)
                for (int i = 0; i < BJ; ++i) {                 // (unrolled, 256 entries are 64 copies a lane and stage, by 4 bytes 256)
                    const int j = h % BCOLS + i * 32, e = j % (BCOLS / 2) * BU;
                    const bool is_c = j >= BCOLS / 2, in_e = e < a.states;
                    const float* src = (is_c ? a.C : a.B) + (size_t)(begin + t0) * a.bc_t + (in_e ? e : 0);
                    float* d = st + 3 * L::ROWS + e / E * 2 * E + (is_c ? E : 0) + e % E;
#pragma unroll
                    for (int k = 0; k < STAGE / BT; ++k) {
                        const int t = (BCOLS <= 32 ? b0 : 0) + k * BT;
                        const bool in = t < nt && in_e;
                        ss_copy<BU * 4>(d + t * 2 * P, src + (long)(in ? t : 0) * bc_t, in);
                    }
                }
            }
        };
        for (int s = 0; s < 3; ++s) copy_stage(s);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();                                       // stages 0, 1 and 2 are in
        __syncthreads();
        for (int s = 0; s < stages; ++s) {
            copy_stage(s + 3);                                 // into the place of stage s - 2, whose outputs are made
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
        }
        return;
    }

    if (tid < SS_WALKERS<G> + 160) {
        // the step sizes of a stage, and its gates in the place of z; a token past the end has step size 0: decay 1 and nothing added
        constexpr int PER = 128 / CH, OWN = (STAGE + PER - 1) / PER;
        const int h = tid - SS_WALKERS<G> - 32, lc = h % CH, own = h / CH, c = c0 + lc;
        const float bias = a.dt_bias[c < a.inner ? c : 0];
        auto prepare = [&](int s) {
            float* st = ss_smem + (s % L::STAGES) * L::STAGE_FLOATS + lc;
            unsigned char* to = steps + (s % 3 * CH + lc) * L::STEP_PITCH;
#pragma unroll
            for (int o = 0; o < OWN; ++o) {
                const int t = o * PER + own;
                if (STAGE % PER && t >= STAGE) break;
                const ACC dt = ss_softplus((ACC)(st[t * CH + L::ROWS] + bias));
                const ACC mine = s * STAGE + t < n ? dt : (ACC)0;
                ss_put2(to + t * 2 * sizeof(ACC), mine, mine * (ACC)st[t * CH]);
                if (gated) st[t * CH + 2 * L::ROWS] = ss_gate(st[t * CH + 2 * L::ROWS], ACC());
            }
        };
        __syncthreads();
        prepare(0);
        prepare(1);
        __syncthreads();
        for (int s = 0; s < stages; ++s) {
            prepare(s + 2);                                    // past the last stage: of stale rows, and nobody uses it
            __syncthreads();
        }
        return;
    }

    // the outputs of the stage behind: a thread takes a channel's run and adds up its lanes' sums
    constexpr int ITEMS = CH * (STAGE / RUN), OWN = (ITEMS + 63) / 64;
    const int h = tid - SS_WALKERS<G> - 160, lc = h % CH, c = c0 + lc;
    const bool ok = c < a.inner;
    const float Dc = a.D[ok ? c : 0];
    T* out = reinterpret_cast<T*>(a.out) + (size_t)begin * a.out_t + (ok ? c : 0);
    auto finish = [&](int s) {
        const float* st = ss_smem + (s % L::STAGES) * L::STAGE_FLOATS + lc;
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
            const int run = h / CH + o * (64 / CH);
            if (ITEMS % 64 && run >= STAGE / RUN) break;
            ACC y[RUN];
            ss_gather<G, RUN>(sums + (s & 1) * L::SUM_BYTES + (run * CH + lc) * L::SUM_PITCH, y);
            const int t0 = run * RUN, at = s * STAGE + t0;
            T* to = out + (size_t)at * a.out_t;
#pragma unroll
            for (int t = 0; t < RUN; ++t) {
                float v = (float)fma((ACC)Dc, (ACC)st[(t0 + t) * CH], y[t]);
                if (gated) v *= st[(t0 + t) * CH + 2 * L::ROWS];
                if (ok && at + t < n) to[t * a.out_t] = from_float<T>(v);
            }
        }
    };
    __syncthreads();
    __syncthreads();
    for (int s = 0; s < stages; ++s) {
        if (s > 0) finish(s - 1);
        __syncthreads();
    }
    finish(stages - 1);
}

template <typename T, typename ACC, int G, int E>
void launch_scan(const ScanArgs& a, int max_q_len, cudaStream_t stream) {
    constexpr int CH = SS_WALKERS<G> / G, U = E < 4 ? E : 4;      // channels of a block, in both forms
    const int R = a.requests;
    const dim3 grid((unsigned)((a.inner + CH - 1) / CH * R));
    if (max_q_len == 1 || a.singles) llmp_launch_dependent(selective_step_kernel<T, ACC, G, E>, grid, dim3(SS_WALKERS<G>), 0, stream, a);
    if (max_q_len == 1) return;
    const bool wide = a.inner % CH == 0 && ((uintptr_t)a.x | (uintptr_t)a.dt | (uintptr_t)a.z) % 16 == 0 && (a.x_t | a.dt_t | a.z_t) % 4 == 0 &&
                      a.states == G * E && ((uintptr_t)a.B | (uintptr_t)a.C) % (4 * U) == 0 && a.bc_t % U == 0 && (a.x_t | a.dt_t | a.z_t | a.bc_t) < (1l << 31);
    constexpr size_t smem = ScanSmem<ACC, G, E>::BYTES;
    auto launch = [&](auto kernel) { llmp_launch_dependent(kernel, grid, dim3(SS_WALKERS<G> + 224), smem, stream, a); };
    if (wide) {
        LLMP_ALLOW_SMEM((selective_walk_kernel<T, ACC, G, E, true>), smem);
        launch(selective_walk_kernel<T, ACC, G, E, true>);
    } else {
        LLMP_ALLOW_SMEM((selective_walk_kernel<T, ACC, G, E, false>), smem);
        launch(selective_walk_kernel<T, ACC, G, E, false>);
    }
}

template <int G, int E> int launch_scan(const ScanArgs& a, int out_dtype, int max_q_len, cudaStream_t stream) {
    constexpr int CH = SS_WALKERS<G> / G;
    LLMP_REQUIRE(((long)a.inner + CH - 1) / CH * a.requests < (1l << 31), "selective_scan: too many channels %d of %d requests", a.inner, a.requests);
    if (out_dtype == LLMP_BF16) launch_scan<bf16, float, G, E>(a, max_q_len, stream);
    else launch_scan<float, double, G, E>(a, max_q_len, stream);
    return llmp_check_launch("selective_scan");
}

// ---- few channels and many tokens: segments side by side ---------------------------------------------------------------
// The recurrence is linear in S, and over a run of tokens every entry decays by exp(A times the sum of the step sizes). So a
// request's tokens are cut into segments of SEG_TOKENS, counted from the portion's first token, and three launches take them:
//   1. every segment but a request's last, from a zero state: its own sum and the sum of its step sizes, to scratch;
//   2. along a request's segments: scratch becomes the state before each (requests of one segment have nothing to do);
//   3. every segment from the state before it: the outputs; the last segment leaves the state in the slot.
// This takes every exponential twice, but nothing waits for a chain of all tokens: where the channels are too few to fill the chip
// and the tokens many, it ends first. The caller draws the line (`scan_prefers_segments`): 4,096 tokens of 16 entries, walk against
// segments, 512 channels 103 and 64 us, 1,024 104 and 92, 2,048 136 and 127, 4,096 184 and 226.
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
    a.slots = slots; a.positions = positions; a.out = out; a.out_t = out_t; a.inner = inner; a.states = states;
    g.sums = entries ? scratch : nullptr; g.steps = scratch + entries * inner * padded; g.requests = R;
    const int segments = more + R;
    if (padded == 8) launch_segments<8>(g, segments, stream);
    else if (padded == 16) launch_segments<16>(g, segments, stream);
    else launch_segments<32>(g, segments, stream);
    return llmp_check_launch("selective_scan_segments");
}

// max_q_len: the most tokens a request brings, or more. singles: 1 where a request of this step may bring a single token beside longer ones
// (0 costs such a request the walk, with the same bits, and saves the others a launch). held: 1 where A, D and dt_bias are
// the caller's for good, so that they may be read while the kernel before is still at work.
LLMP_API int llmp_selective_scan(const float* x, long x_t, const float* dt, long dt_t, const float* dt_bias, const float* B,
                                 const float* C, long bc_t, const float* A, const float* D, const float* z, long z_t, float* state,
                                 long state_slot, long state_half, const int* q_start, const int* slots, const int* positions,
                                 void* out, int out_dtype, long out_t, int R, int inner, int states, int max_q_len, int singles, int held, cudaStream_t stream) {
    if (R <= 0) return 0;
    LLMP_REQUIRE(inner > 0 && states > 0 && states <= 256, "selective_scan: %d channels with %d state entries (up to 256 are served)",
                 inner, states);
    LLMP_REQUIRE(state_half >= (long)inner * states, "selective_scan: the state piece is shorter than the state");
    ScanArgs a;
    a.x = x; a.x_t = x_t; a.dt = dt; a.dt_t = dt_t; a.dt_bias = dt_bias; a.B = B; a.C = C; a.bc_t = bc_t; a.A = A; a.D = D;
    a.z = z; a.z_t = z ? z_t : 0; a.state = state; a.state_slot = state_slot; a.state_half = state_half; a.q_start = q_start;
    a.slots = slots; a.positions = positions; a.out = out; a.out_t = out_t; a.inner = inner; a.states = states;
    a.requests = R; a.singles = singles && R > 1; a.held = held;
    if (states <= 8) return launch_scan<4, 2>(a, out_dtype, max_q_len, stream);
    if (states <= 16) return launch_scan<8, 2>(a, out_dtype, max_q_len, stream);
    if (states <= 32) return launch_scan<16, 2>(a, out_dtype, max_q_len, stream);
    if (states <= 64) return launch_scan<32, 2>(a, out_dtype, max_q_len, stream);
    if (states <= 128) return launch_scan<32, 4>(a, out_dtype, max_q_len, stream);
    return launch_scan<32, 8>(a, out_dtype, max_q_len, stream);
}
