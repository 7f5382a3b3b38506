// Selective scan (Mamba) with its short causal convolution, over segments of consecutive tokens of many sequences.
//
//   xc = silu(conv(x) + b)                              (per channel, `taps` inputs back)
//   S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c xc_c B_n      dt_c = softplus(dt_raw_c + dt_b_c)
//   y_c = (sum_n S[c, n] C_n + D_c xc_c) * silu(z_c)
//
// The recurrent state S and everything that enters it is fp32; x, z and y are activations (bf16 or f32).  A sequence's
// state lives in a slot: S and the last taps - 1 inputs of the convolution.  A segment that starts at position 0 starts from
// zeros whatever the slot holds, so a slot needs no clearing when a new sequence takes it.
//
// Prompts: a CTA owns 16 channels of one segment and walks its tokens in tiles of 32 that cp.async brings into a two-stage
// ring; eight threads share a channel's states, so that the chain of dependent steps is one FMA per state and the partial
// sums of eight tokens are exchanged with seven shuffles; where that fills the chip more than twice, fewer threads walk
// (scan_wide_kernel).  Decode: one thread per channel and sequence, eight sequences per
// CTA; the states are requested first and arrive while the step sizes (a small projection) are computed.
//
// Layout of S and A: planes of four states, [plane][channel][4], so that neighbouring threads - channels - read neighbouring
// 16-byte vectors.
#include "decoder_ops.cuh"
#include "mma_utils.cuh"
#include "tc_utils.cuh"
#include <math.h>
#include <algorithm>
#include <type_traits>

namespace jsm {

using tc::smem_u32;

constexpr int SC_CH = 16;       // channels per CTA
constexpr int SC_SUB = 8;       // threads per channel (prompts)
constexpr int SC_THREADS = SC_CH * SC_SUB;
constexpr int SC_TT = 32;       // tokens per tile
constexpr int ST_WARPS = 4;     // decode step: a warp per sequence
constexpr int ST_CH = 32;       // channels per CTA: a lane each
constexpr int ST_THREADS = ST_CH * ST_WARPS;
constexpr int ST_BB = 8;        // sequences per CTA
__host__ __device__ inline long long plane_index(int n, int c, int ip) { return ((long long)(n >> 2) * ip + c) * 4 + (n & 3); }

__device__ __forceinline__ float softplus_f(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
template <typename T>
__device__ __forceinline__ float decay(float x);  // e^x for x <= 0
template <>
__device__ __forceinline__ float decay<float>(float x) { return expf(x); }
template <>
__device__ __forceinline__ float decay<__nv_bfloat16>(float x) { return fast_ex2(LOG2E * x); }
// the forms of a bf16 model: fp32 arithmetic with the fast exponential and logarithm; ln(1 + e) by its series where 1 + e
// would round e away
template <typename T>
__device__ __forceinline__ float softplus_t(float x) {
    if constexpr (sizeof(T) == 4) return softplus_f(x);
    const float e = fast_ex2(LOG2E * x);
    const float series = e * (1.0f - e * (0.5f - e * (0.33333333f - e * (0.25f - e * 0.2f))));
    return x > 20.0f ? x : x < -3.0f ? series : __logf(1.0f + e);
}
template <typename T>
__device__ __forceinline__ float silu_t(float x) {
    if constexpr (sizeof(T) == 4) return silu_f(x);
    return x * fast_rcp(1.0f + fast_ex2(-LOG2E * x));
}

template <typename T>
struct Vec8;
template <>
struct Vec8<float> {
    struct Raw { float4 a, b; };
    __device__ static Raw fetch(const float* p) { return Raw{reinterpret_cast<const float4*>(p)[0], reinterpret_cast<const float4*>(p)[1]}; }
    __device__ static void widen(const Raw& r, float (&v)[8]) {
        v[0] = r.a.x; v[1] = r.a.y; v[2] = r.a.z; v[3] = r.a.w; v[4] = r.b.x; v[5] = r.b.y; v[6] = r.b.z; v[7] = r.b.w;
    }
    __device__ static void load(const float* p, float (&v)[8]) {
        const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    __device__ static void load_old(const float* p, float (&v)[8]) {
        widen(Raw{load_early(reinterpret_cast<const float4*>(p)), load_early(reinterpret_cast<const float4*>(p) + 1)}, v);
    }
    __device__ static void store(float* p, const float (&v)[8]) {
        reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
};
template <>
struct Vec8<__nv_bfloat16> {
    using Raw = uint4;
    __device__ static Raw fetch(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
    __device__ static void load(const __nv_bfloat16* p, float (&v)[8]) { widen(fetch(p), v); }
    __device__ static void load_old(const __nv_bfloat16* p, float (&v)[8]) { widen(load_early(reinterpret_cast<const uint4*>(p)), v); }
    __device__ static void widen(const uint4& w, float (&v)[8]) {
        v[0] = bf16lo(w.x); v[1] = bf16hi(w.x); v[2] = bf16lo(w.y); v[3] = bf16hi(w.y);
        v[4] = bf16lo(w.z); v[5] = bf16hi(w.z); v[6] = bf16lo(w.w); v[7] = bf16hi(w.w);
    }
    __device__ static void store(__nv_bfloat16* p, const float (&v)[8]) {
        uint4 w;
        w.x = pack_bf16x2(v[0], v[1]); w.y = pack_bf16x2(v[2], v[3]); w.z = pack_bf16x2(v[4], v[5]); w.w = pack_bf16x2(v[6], v[7]);
        *reinterpret_cast<uint4*>(p) = w;
    }
};

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 a = *reinterpret_cast<const uint2*>(p);
    v[0] = bf16lo(a.x); v[1] = bf16hi(a.x); v[2] = bf16lo(a.y); v[3] = bf16hi(a.y);
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
}

// ---- convolution --------------------------------------------------------------------------------------------------
// A thread owns 8 channels of TOK consecutive tokens (8 share the loads of a window; a pass that would leave multiprocessors without
// threads takes 2, a decode step 1); TAPS 0: taps is only known at run time.  carry: every segment is one token, and the state
// moves on by it here (otherwise the scan does that, once every CTA has read the old state)
template <typename T, int TAPS, int TOK>
__global__ void __launch_bounds__(256, 2) scan_conv_kernel(const T* xz, long long pitch, T* xc, T* state,
                                                        const float* __restrict__ w, const float* __restrict__ b,
                                                        const int32_t* __restrict__ seg_start, const int32_t* __restrict__ seg_len,
                                                        const int32_t* __restrict__ seg_pos0, const int32_t* __restrict__ seg_slot, int ip,
                                                        int taps_rt, int carry) {
    // What describes the pass, the constants and the inputs before the segment, kept from earlier passes, are there before the predecessor ends;
    // only the segment's own inputs are waited for (3.9 us a launch in a step of eight sequences, most of it four round trips).
    chain_trigger();
    const int taps = TAPS ? TAPS : taps_rt;
    const int seg = blockIdx.y, vec = ip / 8;
    const int start = load_early(seg_start + seg), len = load_early(seg_len + seg), pos0 = load_early(seg_pos0 + seg);
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int c = (int)(i % vec) * 8, j0 = (int)(i / vec) * TOK;
    if (j0 >= len) return;
    T* st = state + (long long)load_early(seg_slot + seg) * (taps - 1) * ip + c;
    // input of the segment's token j (negative: before the segment)
    auto before = [&](int j, float (&v)[8]) {
        if (pos0 + j >= 0) Vec8<T>::load_old(st + (long long)(taps - 1 + j) * ip, v);
        else
            for (int e = 0; e < 8; ++e) v[e] = 0.0f;
    };
    auto input = [&](int j, float (&v)[8]) {
        if (j >= 0) Vec8<T>::load(xz + (start + j) * pitch + c, v);
        else before(j, v);
    };
    float bias[8];
    if (b) Vec8<float>::load(b + c, bias);
    else
#pragma unroll
        for (int e = 0; e < 8; ++e) bias[e] = 0.0f;
    const int j1 = min(len, j0 + TOK);
    if constexpr (TAPS > 0) {
        float win[TAPS][8], wt[TAPS][8];
#pragma unroll
        for (int k = 0; k < TAPS; ++k) Vec8<float>::load(w + (long long)k * ip + c, wt[k]);
#pragma unroll
        for (int k = 0; k + 1 < TAPS; ++k)
            if (j0 - TAPS + 1 + k < 0) before(j0 - TAPS + 1 + k, win[k + 1]);
        chain_wait();
        // all the thread's inputs are requested before the first is used
        typename Vec8<T>::Raw raw[TOK];
#pragma unroll
        for (int u = 0; u < TOK; ++u)
            if (j0 + u < j1) raw[u] = Vec8<T>::fetch(xz + (start + j0 + u) * pitch + c);
#pragma unroll
        for (int k = 0; k + 1 < TAPS; ++k)
            if (j0 - TAPS + 1 + k >= 0) input(j0 - TAPS + 1 + k, win[k + 1]);
#pragma unroll
        for (int u = 0; u < TOK; ++u) {
            const int j = j0 + u;
            if (j >= j1) break;
#pragma unroll
            for (int k = 0; k + 1 < TAPS; ++k)
#pragma unroll
                for (int e = 0; e < 8; ++e) win[k][e] = win[k + 1][e];
            Vec8<T>::widen(raw[u], win[TAPS - 1]);
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float a = bias[e];
#pragma unroll
                for (int k = 0; k < TAPS; ++k) a = fmaf(wt[k][e], win[k][e], a);
                o[e] = silu_t<T>(a);
            }
            Vec8<T>::store(xc + (long long)(start + j) * ip + c, o);
        }
        if (carry)  // one token per segment: this thread has read all there is to read of its channels' state
#pragma unroll
            for (int k = 0; k + 1 < TAPS; ++k) Vec8<T>::store(st + (long long)k * ip, win[k + 1]);
    } else {
        chain_wait();
        for (int j = j0; j < j1; ++j) {
            float o[8];
            for (int e = 0; e < 8; ++e) o[e] = bias[e];
            for (int k = 0; k < taps; ++k) {
                float v[8], wk[8];
                input(j - taps + 1 + k, v);
                Vec8<float>::load(w + (long long)k * ip + c, wk);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = fmaf(wk[e], v[e], o[e]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = silu_t<T>(o[e]);
            Vec8<T>::store(xc + (long long)(start + j) * ip + c, o);
        }
        if (carry)
            for (int k = 0; k + 1 < taps; ++k) {
                float v[8];
                input(k + 2 - taps, v);  // ascending: an entry is read before a later one takes its place
                Vec8<T>::store(st + (long long)k * ip, v);
            }
    }
}

// the last taps - 1 inputs after the segment: entry k is the input taps - 1 - k tokens before the next one.  One thread per
// channel, ascending k: an entry taken from the old state lies behind every entry already written.
template <typename T>
__device__ __forceinline__ void carry_conv_state(T* state, const T* __restrict__ xz, long long pitch, int c, int ip, int taps, int start, int len,
                                                 int pos0) {
    for (int k = 0; k + 1 < taps; ++k) {
        const int j = len - (taps - 1) + k;
        T v = from_f32<T>(0.0f);
        if (j >= 0) v = xz[(start + j) * pitch + c];
        else if (pos0 + j >= 0) v = state[(long long)(k + len) * ip + c];
        state[(long long)k * ip + c] = v;
    }
}

template <int NS>
__device__ __forceinline__ void lds_vec(const float* p, float (&v)[NS]) {
    if constexpr (NS % 4 == 0) {
#pragma unroll
        for (int i = 0; i < NS; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(p + i);
            v[i] = a.x; v[i + 1] = a.y; v[i + 2] = a.z; v[i + 3] = a.w;
        }
    } else if constexpr (NS % 2 == 0) {
#pragma unroll
        for (int i = 0; i < NS; i += 2) {
            const float2 a = *reinterpret_cast<const float2*>(p + i);
            v[i] = a.x; v[i + 1] = a.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NS; ++i) v[i] = p[i];
    }
}

template <int NS>
__device__ __forceinline__ void lds_pairs(const float* p, uint64_t (&v)[NS / 2]) {
    if constexpr (NS % 4 == 0) {
#pragma unroll
        for (int i = 0; i < NS / 2; i += 2) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(p + 2 * i);
            v[i] = w.x; v[i + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NS / 2; ++i) v[i] = *reinterpret_cast<const uint64_t*>(p + 2 * i);
    }
}

// eight tokens' partial sums on each of SUB lanes -> the sums of tokens 8 / SUB * sub .. in y[0 ..]
template <int SUB>
__device__ __forceinline__ void column_sums(float (&y)[8], int sub) {
#pragma unroll
    for (int w = SUB / 2, m = 4; w >= 1; w >>= 1, m >>= 1) {
        const bool high = sub & w;
#pragma unroll
        for (int u = 0; u < m; ++u) y[u] = (high ? y[m + u] : y[u]) + __shfl_xor_sync(0xffffffffu, high ? y[u] : y[m + u], w);
    }
}

// ---- scan of prompts ----------------------------------------------------------------------------------------------
template <typename T, int NS>
constexpr int scan_smem() {
    return 2 * SC_TT * SC_CH * (2 * (int)sizeof(T) + 4) + 2 * SC_TT * 2 * SC_SUB * NS * 4 + SC_TT * (SC_CH + 4) * 4 + SC_TT * SC_CH * 16;
}

struct ScanArgs {
    const float *A, *D, *dt_b, *proj, *dt_raw;
    const void *xz, *xc, *dt_w;
    void *y, *conv;
    float* S;
    const int32_t *seg_start, *seg_len, *seg_pos0, *seg_slot;
    int ip, np, rp, state, taps, n_segs;
};

// NS states per thread.  The bf16 instance of 9 to 16 states only runs with up to two CTAs per SM (scan_dispatch): a minimum of four gives it 120
// registers instead of 54, and the loads of a group of tokens move ahead (2048 tokens, 2048 channels 118 -> 107 us, 4096 channels 135 -> 127).
template <typename T, int NS>
__global__ void __launch_bounds__(SC_THREADS, sizeof(T) == 2 && NS == 2 ? 4 : 0) scan_kernel(ScanArgs a) {
    extern __shared__ __align__(16) uint8_t sc_dyn[];
    constexpr int CH = SC_CH, SUB = SC_SUB, YP = CH + 4, NB = SUB * NS;     // YP: pitch of the output tile; NB: B / C columns per tile row
    constexpr int EL = SC_TT * CH / SC_THREADS;                             // elements of a tile per thread
    T* xs = reinterpret_cast<T*>(sc_dyn);                                   // 2 x [TT][CH]
    T* zs = xs + 2 * SC_TT * CH;                                         // 2 x [TT][CH]
    float* dts = reinterpret_cast<float*>(zs + 2 * SC_TT * CH);          // 2 x [TT][CH]
    float* bc = dts + 2 * SC_TT * CH;                                    // 2 x [TT][B: NB | C: NB]
    float* ys = bc + 2 * SC_TT * 2 * NB;                                    // [TT][YP]
    float4* dd = reinterpret_cast<float4*>(ys + SC_TT * YP);             // [TT][CH]: dt, dt, dt x, dt x
    constexpr bool PAIRS = sizeof(T) == 2 && NS % 2 == 0;                   // bf16 models: states in pairs, base-2 exponentials
    chain_trigger();
    const int tid = threadIdx.x, ch = tid / SUB, sub = tid % SUB;
    const int c0 = blockIdx.x * CH, c = c0 + ch;
    const bool live = c < a.ip;
    float A[NS], S[NS];
    uint64_t A2[PAIRS ? NS / 2 : 1], S2[PAIRS ? NS / 2 : 1];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        const int n = sub * NS + i;
        A[i] = (live && n < a.state) ? a.A[plane_index(n, c, a.ip)] : 0.0f;
        if (PAIRS) A[i] *= LOG2E;
    }
    for (int i = tid; i < 2 * SC_TT * 2 * NB; i += SC_THREADS) bc[i] = 0.0f;  // columns behind np stay zero
    __syncthreads();
    chain_wait();
    const int seg = blockIdx.y;
    const int start = a.seg_start[seg], len = a.seg_len[seg], pos0 = a.seg_pos0[seg], slot = a.seg_slot[seg];
    float* state = a.S + (long long)slot * a.ip * a.np;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        const int n = sub * NS + i;
        S[i] = (live && n < a.state && pos0 > 0) ? state[plane_index(n, c, a.ip)] : 0.0f;
    }
    if constexpr (PAIRS)
#pragma unroll
        for (int i = 0; i < NS / 2; ++i) { A2[i] = f2_pack(A[2 * i], A[2 * i + 1]); S2[i] = f2_pack(S[2 * i], S[2 * i + 1]); }
    const int pc = a.rp + 2 * a.np;
    const T* xz = static_cast<const T*>(a.xz);
    const T* xc = static_cast<const T*>(a.xc);
    auto load_tile = [&](int t0, int stage) {
        constexpr int EV = 16 / sizeof(T), XV = CH / EV;  // elements per vector, vectors per row
        for (int i = tid; i < SC_TT * XV; i += SC_THREADS) {
            const int r = i / XV, v = (i % XV) * EV;
            const bool ok = t0 + r < len && c0 + v < a.ip;
            const long long t = start + (ok ? t0 + r : 0);
            const int cc = ok ? c0 + v : 0;
            cp_async16(smem_u32(xs + (stage * SC_TT + r) * CH + v), xc + t * a.ip + cc, ok);
            cp_async16(smem_u32(zs + (stage * SC_TT + r) * CH + v), xz + t * 2 * a.ip + a.ip + cc, ok);
        }
        for (int i = tid; i < SC_TT * (CH / 4); i += SC_THREADS) {
            const int r = i / (CH / 4), v = (i % (CH / 4)) * 4;
            const bool ok = t0 + r < len && c0 + v < a.ip;
            cp_async16(smem_u32(dts + (stage * SC_TT + r) * CH + v), a.dt_raw + (long long)(start + (ok ? t0 + r : 0)) * a.ip + (ok ? c0 + v : 0), ok);
        }
        for (int i = tid; i < SC_TT * 2 * (NB / 4); i += SC_THREADS) {
            const int r = i / (2 * (NB / 4)), part = i / (NB / 4) & 1, v = i % (NB / 4) * 4;
            if (v >= a.np) continue;
            const bool ok = t0 + r < len;
            const float* src = a.proj + (long long)(start + (ok ? t0 + r : 0)) * pc + a.rp + part * a.np + v;
            cp_async16(smem_u32(bc + ((stage * SC_TT + r) * 2 + part) * NB + v), src, ok);
        }
    };
    load_tile(0, 0);
    cp_async_commit();
    // every pass over a tile gives a thread the same channels: their constants stay in registers
    static_assert(SC_THREADS % CH == 0 && EL == 4, "four elements of a tile per thread");
    const float bias = c0 + (tid & (CH - 1)) < a.ip ? a.dt_b[c0 + (tid & (CH - 1))] : 0.0f;
    const int ov = (tid & (CH / 4 - 1)) * 4, orow = tid / (CH / 4);  // output pass: four channels of one token
    const bool olive = c0 + ov < a.ip;
    const float4 Dv = olive ? *reinterpret_cast<const float4*>(a.D + c0 + ov) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int nt = (len + SC_TT - 1) / SC_TT;
    for (int it = 0; it < nt; ++it) {
        const int stage = it & 1, t0 = it * SC_TT, n = min(SC_TT, len - t0);
        if (it + 1 < nt) load_tile(t0 + SC_TT, stage ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const float* dt = dts + stage * SC_TT * CH;
        const T* x = xs + stage * SC_TT * CH;
#pragma unroll
        for (int u = 0; u < EL; ++u) {
            const int i = u * SC_THREADS + tid;
            // a step size of zero leaves the state as it is: the rows behind the segment (and channels behind the last)
            const float d = i / CH < n ? softplus_t<T>(dt[i] + bias) : 0.0f, dx = d * to_f32(x[i]);
            dd[i] = make_float4(d, d, dx, dx);
        }
        __syncthreads();
        const float* bt = bc + stage * SC_TT * 2 * NB + sub * NS;
#pragma unroll 1
        for (int t8 = 0; t8 < n; t8 += 8) {
            float y[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t8 + u;
                if constexpr (PAIRS) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(dd + t * CH + ch);  // (dt, dt), (dt x, dt x)
                    uint64_t B[NS / 2], C[NS / 2];
                    lds_pairs<NS>(bt + t * 2 * NB, B);
                    lds_pairs<NS>(bt + t * 2 * NB + NB, C);
                    uint64_t acc = 0;
#pragma unroll
                    for (int i = 0; i < NS / 2; ++i) {
                        float e0, e1;
                        f2_unpack(f2_mul(w.x, A2[i]), e0, e1);
                        S2[i] = f2_fma(f2_pack(fast_ex2(e0), fast_ex2(e1)), S2[i], f2_mul(w.y, B[i]));
                        acc = i == 0 ? f2_mul(S2[i], C[i]) : f2_fma(S2[i], C[i], acc);
                    }
                    float lo, hi;
                    f2_unpack(acc, lo, hi);
                    y[u] = lo + hi;
                } else {
                    const float4 w = dd[t * CH + ch];
                    float B[NS], C[NS];
                    lds_vec<NS>(bt + t * 2 * NB, B);
                    lds_vec<NS>(bt + t * 2 * NB + NB, C);
                    float acc = 0.0f;
#pragma unroll
                    for (int i = 0; i < NS; ++i) {
                        S[i] = fmaf(decay<T>(w.x * A[i]), S[i], w.z * B[i]);
                        acc = fmaf(S[i], C[i], acc);
                    }
                    y[u] = acc;
                }
            }
            column_sums<SUB>(y, sub);
            ys[(t8 + sub) * YP + ch] = y[0];
        }
        __syncthreads();
        const T* z = zs + stage * SC_TT * CH;
        if (orow < n && olive) {
            float xv[4], zv[4], o[4];
            load4(x + orow * CH + ov, xv);
            load4(z + orow * CH + ov, zv);
            const float4 yv = *reinterpret_cast<const float4*>(ys + orow * YP + ov);
            o[0] = fmaf(Dv.x, xv[0], yv.x) * silu_t<T>(zv[0]); o[1] = fmaf(Dv.y, xv[1], yv.y) * silu_t<T>(zv[1]);
            o[2] = fmaf(Dv.z, xv[2], yv.z) * silu_t<T>(zv[2]); o[3] = fmaf(Dv.w, xv[3], yv.w) * silu_t<T>(zv[3]);
            store4(static_cast<T*>(a.y) + (long long)(start + t0 + orow) * a.ip + c0 + ov, o);
        }
        __syncthreads();
    }
    if constexpr (PAIRS)
#pragma unroll
        for (int i = 0; i < NS / 2; ++i) f2_unpack(S2[i], S[2 * i], S[2 * i + 1]);
    if (live)
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if (sub * NS + i < a.state) state[plane_index(sub * NS + i, c, a.ip)] = S[i];
    if (tid < CH && c0 + tid < a.ip)
        carry_conv_state(static_cast<T*>(a.conv) + (long long)slot * (a.taps - 1) * a.ip, xz, 2 * a.ip, c0 + tid, a.ip, a.taps, start, len,
                            pos0);
}

// ---- scan of prompts, bf16 models with 9 to 16 states, chip filled --------------------------------------------------
// What bounds it: instructions, then exponentials.  In scan_kernel above the exchange of partial sums, the broadcast of step
// sizes as pairs and the passes over a tile cost as much as the states themselves (33 instructions per warp and token, the
// issue slots of the fullest SMs 72 % in use).  Here two threads share a channel, eight states each, so that a token costs half the
// instructions per state and one exchange per eight tokens and channel; and four warps that do nothing else walk the tokens,
// one per scheduler, the decays of a token computed while the one before it moves the state.  Four more warps bring the
// tiles, make the step sizes of the next one and write the outputs of the last one meanwhile.  A CTA owns 64 channels.
// 2048 tokens, 16 states, 8192 channels: 224 -> 139 us with cold caches (scan_kernel 194, where addresses with constant strides and states kept as pairs save a
// seventh); the exponential units are then three quarters in use on the 128 SMs that have a CTA.  With sums in an order of their own, warm 131 us: eight walking warps of
// four states 148 us, eight warps beside the walking ones 156; 2 CTAs per SM are named because the compiler then takes 126 registers, without that 66 (165 us).
constexpr int SW_CH = 64, SW_SUB = 2, SW_NS = 8, SW_HELP = 128, SW_MAIN = SW_CH * SW_SUB, SW_THREADS = SW_MAIN + SW_HELP, SW_YP = SW_CH + 4;
struct ScanWideTile {  // a tile as it arrives
    __nv_bfloat16 x[SC_TT][SW_CH], z[SC_TT][SW_CH];
};
struct ScanWideShared {
    ScanWideTile in[3];
    float bc[3][SC_TT + 2][2][SW_SUB * SW_NS];  // (two rows more: what is fetched ahead behind a tile's end is not used)
    float raw[2][SC_TT][SW_CH];   // step sizes before the softplus
    float2 dd[2][SC_TT + 2][SW_CH];  // dt, dt x
    float y[2][SC_TT][SW_YP];
};
// A token's sum over the states is formed in the order of scan_kernel, so that a prompt's outputs do not depend on which of the two runs: there thread k
// adds states 2 k and 2 k + 1, and eight such pairs meet in exchanges of distance 4, 2 and 1.  So a thread here has the pairs sub, sub + 2, sub + 4
// and sub + 6, the even and the odd states of two pairs packed: element e of register i is state sw_state(sub, i, e), which lies at sw_place.
__device__ __forceinline__ int sw_state(int sub, int i, int e) { return 2 * (sub + 2 * e + 4 * (i >> 1)) + (i & 1); }
__device__ __forceinline__ int sw_place(int n) { return (n >> 1 & 1) * SW_NS + (n >> 3) * 4 + (n & 1) * 2 + (n >> 2 & 1); }

__global__ void __launch_bounds__(SW_THREADS, 2) scan_wide_kernel(ScanArgs a) {
    extern __shared__ __align__(16) uint8_t sc_dyn[];
    ScanWideShared& sh = *reinterpret_cast<ScanWideShared*>(sc_dyn);
    constexpr int NS = SW_NS, NB = SW_SUB * NS;
    chain_trigger();
    const int tid = threadIdx.x, c0 = blockIdx.x * SW_CH, seg = blockIdx.y;
    chain_wait();
    const int start = a.seg_start[seg], len = a.seg_len[seg], pos0 = a.seg_pos0[seg], slot = a.seg_slot[seg];
    const int nt = (len + SC_TT - 1) / SC_TT;
    if (tid >= SW_MAIN) {
        const int h = tid - SW_MAIN, pc = a.rp + 2 * NB;  // (9 to 16 states are kept as 16)
        const __nv_bfloat16 *xz = static_cast<const __nv_bfloat16*>(a.xz), *xc = static_cast<const __nv_bfloat16*>(a.xc);
        auto load = [&](int it) {
            const int t0 = it * SC_TT, b3 = it % 3;
            ScanWideTile& in = sh.in[b3];
#pragma unroll
            for (int u = 0; u < SC_TT * (SW_CH / 8) / SW_HELP; ++u) {
                const int r = (h + u * SW_HELP) / (SW_CH / 8), v = (h + u * SW_HELP) % (SW_CH / 8) * 8;
                const bool ok = t0 + r < len && c0 + v < a.ip;
                const long long t = start + (ok ? t0 + r : 0);
                const int cc = ok ? c0 + v : 0;
                cp_async16(smem_u32(&in.x[r][v]), xc + t * a.ip + cc, ok);
                cp_async16(smem_u32(&in.z[r][v]), xz + t * 2 * a.ip + a.ip + cc, ok);
            }
#pragma unroll
            for (int u = 0; u < SC_TT * (SW_CH / 4) / SW_HELP; ++u) {
                const int r = (h + u * SW_HELP) / (SW_CH / 4), v = (h + u * SW_HELP) % (SW_CH / 4) * 4;
                const bool ok = t0 + r < len && c0 + v < a.ip;
                cp_async16(smem_u32(&sh.raw[it & 1][r][v]), a.dt_raw + (long long)(start + (ok ? t0 + r : 0)) * a.ip + (ok ? c0 + v : 0), ok);
            }
#pragma unroll
            for (int u = 0; u < SC_TT * 2 * NB / SW_HELP; ++u) {
                const int r = h / (2 * NB) + u * (SW_HELP / (2 * NB)), part = h / NB & 1, n = h % NB;
                const bool ok = t0 + r < len;
                cp_async4(smem_u32(&sh.bc[b3][r][part][sw_place(n)]), a.proj + (long long)(start + (ok ? t0 + r : 0)) * pc + a.rp + part * NB + n, ok);
            }
            cp_async_commit();
        };
        const int ov = h % (SW_CH / 4) * 4, row0 = h / (SW_CH / 4);  // four channels of every eighth token
        const bool olive = c0 + ov < a.ip;
        const float4 bias = olive ? *reinterpret_cast<const float4*>(a.dt_b + c0 + ov) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 D = olive ? *reinterpret_cast<const float4*>(a.D + c0 + ov) : make_float4(0.f, 0.f, 0.f, 0.f);
        auto step_sizes = [&](int it) {
            const int n = len - it * SC_TT;
#pragma unroll
            for (int r = row0; r < SC_TT; r += SW_HELP / (SW_CH / 4)) {
                // a step size of zero leaves the state as it is: the rows behind the segment
                const float4 w = *reinterpret_cast<const float4*>(&sh.raw[it & 1][r][ov]);
                float x[4], d[4] = {softplus_t<__nv_bfloat16>(w.x + bias.x), softplus_t<__nv_bfloat16>(w.y + bias.y),
                                    softplus_t<__nv_bfloat16>(w.z + bias.z), softplus_t<__nv_bfloat16>(w.w + bias.w)};
                load4(&sh.in[it % 3].x[r][ov], x);
                if (r >= n) d[0] = d[1] = d[2] = d[3] = 0.0f;
                float4* o = reinterpret_cast<float4*>(&sh.dd[it & 1][r][ov]);
                o[0] = make_float4(d[0], d[0] * x[0], d[1], d[1] * x[1]);
                o[1] = make_float4(d[2], d[2] * x[2], d[3], d[3] * x[3]);
            }
        };
        auto outputs = [&](int it) {
            const int t0 = it * SC_TT, n = min(SC_TT, len - t0);
            if (!olive) return;
#pragma unroll
            for (int r = row0; r < SC_TT; r += SW_HELP / (SW_CH / 4)) {
                if (r >= n) break;
                float xv[4], zv[4], o[4];
                load4(&sh.in[it % 3].x[r][ov], xv);
                load4(&sh.in[it % 3].z[r][ov], zv);
                const float4 y = *reinterpret_cast<const float4*>(&sh.y[it & 1][r][ov]);
                o[0] = fmaf(D.x, xv[0], y.x) * silu_t<__nv_bfloat16>(zv[0]); o[1] = fmaf(D.y, xv[1], y.y) * silu_t<__nv_bfloat16>(zv[1]);
                o[2] = fmaf(D.z, xv[2], y.z) * silu_t<__nv_bfloat16>(zv[2]); o[3] = fmaf(D.w, xv[3], y.w) * silu_t<__nv_bfloat16>(zv[3]);
                store4(static_cast<__nv_bfloat16*>(a.y) + (long long)(start + t0 + r) * a.ip + c0 + ov, o);
            }
        };
        auto helpers_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(SW_HELP) : "memory"); };
        load(0);
        if (nt > 1) load(1);
        if (nt > 1) cp_async_wait<1>();
        else cp_async_wait<0>();
        helpers_sync();
        step_sizes(0);
        __syncthreads();
        for (int it = 0; it < nt; ++it) {
            if (it > 0) outputs(it - 1);
            if (it + 1 < nt) {
                cp_async_wait<0>();
                helpers_sync();  // tile it + 1 is there; nobody reads tile it - 1 any more
                if (it + 2 < nt) load(it + 2);
                step_sizes(it + 1);
            }
            __syncthreads();
        }
        if (nt > 0) outputs(nt - 1);
        if (h < SW_CH && c0 + h < a.ip)
            carry_conv_state(static_cast<__nv_bfloat16*>(a.conv) + (long long)slot * (a.taps - 1) * a.ip, xz, 2 * a.ip, c0 + h, a.ip, a.taps, start, len, pos0);
        return;
    }
    const int ch = tid / SW_SUB, sub = tid % SW_SUB, c = c0 + ch;
    const bool live = c < a.ip;
    float* state = a.S + (long long)slot * a.ip * NB;
    uint64_t A[NS / 2], S[NS / 2];
#pragma unroll
    for (int i = 0; i < NS / 2; ++i) {
        float p[2], q[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = sw_state(sub, i, e);
            p[e] = live && n < a.state ? a.A[plane_index(n, c, a.ip)] * LOG2E : 0.0f;
            q[e] = live && n < a.state && pos0 > 0 ? state[plane_index(n, c, a.ip)] : 0.0f;
        }
        A[i] = f2_pack(p[0], p[1]);
        S[i] = f2_pack(q[0], q[1]);
    }
    __syncthreads();
    for (int it = 0; it < nt; ++it) {
        const int n = min(SC_TT, len - it * SC_TT), b3 = it % 3, b2 = it & 1;
        float2 w[4];
        uint64_t B[2][NS / 2], C[2][NS / 2], decay[2][NS / 2];
        auto fetch = [&](int t, int x) {
            lds_pairs<NS>(&sh.bc[b3][t][0][sub * NS], B[x & 1]);
            lds_pairs<NS>(&sh.bc[b3][t][1][sub * NS], C[x & 1]);
        };
        auto decays = [&](int x) {
            const uint64_t dt = f2_pack(w[x & 3].x, w[x & 3].x);
#pragma unroll
            for (int i = 0; i < NS / 2; ++i) {
                float e0, e1;
                f2_unpack(f2_mul(dt, A[i]), e0, e1);
                decay[x & 1][i] = f2_pack(fast_ex2(e0), fast_ex2(e1));
            }
        };
        w[0] = sh.dd[b2][0][ch];
        w[1] = sh.dd[b2][1][ch];
        fetch(0, 0);
        decays(0);
#pragma unroll 1
        for (int t8 = 0; t8 < n; t8 += 8) {
            float y[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                fetch(t8 + u + 1, u + 1);
                w[(u + 2) & 3] = sh.dd[b2][t8 + u + 2][ch];
                decays(u + 1);
                const uint64_t dx = f2_pack(w[u & 3].y, w[u & 3].y);
                uint64_t part[NS / 2];
#pragma unroll
                for (int i = 0; i < NS / 2; ++i) {
                    S[i] = f2_fma(decay[u & 1][i], S[i], f2_mul(dx, B[u & 1][i]));
                    part[i] = f2_mul(S[i], C[u & 1][i]);
                }
                // (apart: a packed product whose only use is a packed sum becomes an FMA, which does not round the product)
                float p[NS / 2][2];
#pragma unroll
                for (int i = 0; i < NS / 2; ++i) f2_unpack(part[i], p[i][0], p[i][1]);
                y[u] = ((p[0][0] + p[1][0]) + (p[2][0] + p[3][0])) + ((p[0][1] + p[1][1]) + (p[2][1] + p[3][1]));
            }
            column_sums<SW_SUB>(y, sub);
#pragma unroll
            for (int u = 0; u < 8 / SW_SUB; ++u) sh.y[b2][t8 + 8 / SW_SUB * sub + u][ch] = y[u];
        }
        __syncthreads();
    }
    if (live)
#pragma unroll
        for (int i = 0; i < NS / 2; ++i) {
            float p[2];
            f2_unpack(S[i], p[0], p[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (sw_state(sub, i, e) < a.state) state[plane_index(sw_state(sub, i, e), c, a.ip)] = p[e];
        }
}

// ---- decode step --------------------------------------------------------------------------------------------------
// One token of up to 8 sequences and 32 channels per CTA: lane = channel, a warp takes two sequences; the convolution has
// already moved its state on.  The step sizes of the 32 channels x 8 sequences are one small product: bf16 models take it on
// the tensor cores (weights as the 16-row operand, two tiles of channels x two halves of the rank over the four warps).
// NP: planes of four states kept in registers, requested before the step sizes are known; 0 = any number, read when needed.
template <typename T, int NP>
__global__ void __launch_bounds__(ST_THREADS) scan_step_kernel(ScanArgs a) {
    extern __shared__ __align__(16) float st_dyn[];  // bf16: [8][B: np | C: np]; f32: [8][proj columns]
    __shared__ float dts[2][ST_CH][9];
    constexpr bool MMA = sizeof(T) == 2;
    constexpr int R = ST_BB / ST_WARPS;  // sequences per warp
    chain_trigger();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * ST_CH, c = c0 + lane, cl = min(c, a.ip - 1);
    const bool live = c < a.ip;
    const int s0 = blockIdx.y * ST_BB, nb = min(ST_BB, a.n_segs - s0);
    const int pc = a.rp + 2 * a.np, off = MMA ? a.rp : 0, sc = pc - off;  // columns of proj that go to shared memory
    const int planes = a.np / 4;
    const float4* Ap = reinterpret_cast<const float4*>(a.A) + cl;
    float4 A[NP ? NP : 1];
    if (NP > 0)
#pragma unroll
        for (int i = 0; i < NP; ++i) A[i] = i < planes ? Ap[(long long)i * a.ip] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float bias = a.dt_b[cl], dv = a.D[cl];
    // only this kernel writes the states, and passes are separated by the host: they are requested before the predecessor ends
    float4 S[R][NP ? NP : 1];
    float4* Sp[R];
    bool fresh[R];
    int tok[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int sg = s0 + min(q * ST_WARPS + warp, nb - 1);
        tok[q] = load_early(a.seg_start + sg);
        fresh[q] = load_early(a.seg_pos0 + sg) == 0;
        Sp[q] = reinterpret_cast<float4*>(a.S + (long long)load_early(a.seg_slot + sg) * a.ip * a.np) + cl;
        if (NP > 0)
#pragma unroll
            for (int i = 0; i < NP; ++i)
                S[q][i] = (i < planes && !fresh[q]) ? load_early(Sp[q] + (long long)i * a.ip) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    chain_wait();
    for (int i = tid; i < nb * (sc / 4); i += ST_THREADS) {
        const int b = i / (sc / 4), v = i % (sc / 4);
        cp_async16(smem_u32(st_dyn + i * 4), a.proj + (long long)a.seg_start[s0 + b] * pc + off + v * 4, true);
    }
    cp_async_commit();
    T xv[R], zv[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        xv[q] = static_cast<const T*>(a.xc)[(long long)tok[q] * a.ip + cl];
        zv[q] = static_cast<const T*>(a.xz)[(long long)tok[q] * 2 * a.ip + a.ip + cl];
    }
    if constexpr (MMA) {
        const int mt = warp & 1, kh = warp >> 1, g = lane >> 2, kq = (lane & 3) * 8;
        const int n_blk = (a.rp + 31) / 32, b0 = kh ? (n_blk + 1) / 2 : 0, b1 = kh ? n_blk : (n_blk + 1) / 2;
        const int r0 = c0 + mt * 16 + g;
        const __nv_bfloat16* w0 = static_cast<const __nv_bfloat16*>(a.dt_w) + (long long)min(r0, a.ip - 1) * a.rp;
        const __nv_bfloat16* w1 = static_cast<const __nv_bfloat16*>(a.dt_w) + (long long)min(r0 + 8, a.ip - 1) * a.rp;
        const float* p = a.proj + (long long)a.seg_start[s0 + min(g, nb - 1)] * pc;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int blk = b0; blk < b1; ++blk) {
            const int k = blk * 32 + kq;
            uint4 x = make_uint4(0, 0, 0, 0), y = x;
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
            if (k < a.rp) {
                x = __ldg(reinterpret_cast<const uint4*>(w0 + k));
                y = __ldg(reinterpret_cast<const uint4*>(w1 + k));
                u = reinterpret_cast<const float4*>(p + k)[0];
                v = reinterpret_cast<const float4*>(p + k)[1];
            }
            const uint32_t a0[4] = {x.x, y.x, x.y, y.y}, a1[4] = {x.z, y.z, x.w, y.w};
            mma_16816(acc, a0, pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w));
            mma_16816(acc, a1, pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
        }
        float* d = &dts[kh][mt * 16 + g][(lane & 3) * 2];
        d[0] = acc[0]; d[1] = acc[1]; d[8 * 9] = acc[2]; d[8 * 9 + 1] = acc[3];
    }
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int b = q * ST_WARPS + warp;
        if (b >= nb) break;
        float raw = 0.0f;
        if constexpr (MMA) {
            raw = dts[0][lane][b] + dts[1][lane][b];
        } else {
            const T* w = static_cast<const T*>(a.dt_w) + (long long)cl * a.rp;
            for (int r = 0; r < a.rp; ++r) raw = fmaf(to_f32(w[r]), st_dyn[b * sc + r], raw);
        }
        const float x = to_f32(xv[q]), dt = softplus_t<T>(raw + bias), dx = dt * x;
        const float4* Bp = reinterpret_cast<const float4*>(st_dyn + b * sc + (a.rp - off));
        const float4* Cp = Bp + planes;
        float y = 0.0f;
        auto plane = [&](int i, const float4& Ai, float4& s) {
            const float4 B = Bp[i], C = Cp[i];
            s.x = fmaf(decay<T>(dt * Ai.x), s.x, dx * B.x); y = fmaf(s.x, C.x, y);
            s.y = fmaf(decay<T>(dt * Ai.y), s.y, dx * B.y); y = fmaf(s.y, C.y, y);
            s.z = fmaf(decay<T>(dt * Ai.z), s.z, dx * B.z); y = fmaf(s.z, C.z, y);
            s.w = fmaf(decay<T>(dt * Ai.w), s.w, dx * B.w); y = fmaf(s.w, C.w, y);
            if (live) Sp[q][(long long)i * a.ip] = s;
        };
        if constexpr (NP > 0) {
#pragma unroll
            for (int i = 0; i < NP; ++i)
                if (i < planes) plane(i, A[i], S[q][i]);
        } else {
#pragma unroll 2
            for (int i = 0; i < planes; ++i) {
                float4 s = fresh[q] ? make_float4(0.f, 0.f, 0.f, 0.f) : Sp[q][(long long)i * a.ip];
                plane(i, Ap[(long long)i * a.ip], s);
            }
        }
        if (live) static_cast<T*>(a.y)[(long long)tok[q] * a.ip + c] = from_f32<T>(fmaf(dv, x, y) * silu_t<T>(to_f32(zv[q])));
    }
}

__global__ void __launch_bounds__(256) scan_dt_operand_kernel(const float* __restrict__ proj, __nv_bfloat16* __restrict__ out, int T, int rp, int pc) {
    chain_trigger();
    chain_wait();
    const int vec = rp / 8;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < (long long)T * vec; i += (long long)gridDim.x * 256) {
        const int t = (int)(i / vec), c = (int)(i % vec) * 8;
        float v[8];
        Vec8<float>::load(proj + (long long)t * pc + c, v);
        Vec8<__nv_bfloat16>::store(out + (long long)t * rp + c, v);
    }
}

// ---- launches -----------------------------------------------------------------------------------------------------
template <typename T>
static jsm_status conv_typed(const void* x, long long pitch, int cp, int taps, const float* w, const float* b, void* state, const StepTokens& tk, void* out,
                             bool carry, cudaStream_t st) {
    auto run = [&](auto tok) -> jsm_status {
        constexpr int TOK = decltype(tok)::value;
        const long long n = (long long)((tk.max_len + TOK - 1) / TOK) * (cp / 8);
        const dim3 grid((unsigned)((n + 255) / 256), tk.n_segs);
        auto go = [&](auto kernel) {
            return launch_chained(kernel, grid, dim3(256), 0, st, (const T*)x, pitch, (T*)out, (T*)state, w, b, tk.seg_start, tk.seg_len, tk.seg_pos0,
                                  tk.seg_slot, cp, taps, carry ? 1 : 0);
        };
        JSM_CUDA_CHECK(taps == 1 ? go(scan_conv_kernel<T, 1, TOK>) : taps == 2 ? go(scan_conv_kernel<T, 2, TOK>) : taps == 3 ? go(scan_conv_kernel<T, 3, TOK>)
                       : taps == 4 ? go(scan_conv_kernel<T, 4, TOK>) : go(scan_conv_kernel<T, 0, TOK>));
        JSM_LAUNCH_CHECK();
        return JSM_OK;
    };
    if (tk.max_len == 1) return run(std::integral_constant<int, 1>());
    // two CTAs per multiprocessor with eight tokens a thread, else two tokens
    const long long ctas = (long long)((tk.max_len + 7) / 8) * (cp / 8) * tk.n_segs / 256;
    return ctas < 2 * sm_count() ? run(std::integral_constant<int, 2>()) : run(std::integral_constant<int, 8>());
}

jsm_status short_conv_launch(bool f32, const void* x, long long x_pitch, int cp, int taps, const float* w, const float* bias, void* state,
                             const StepTokens& tk, void* out, bool carry, cudaStream_t st) {
    return f32 ? conv_typed<float>(x, x_pitch, cp, taps, w, bias, state, tk, out, carry, st)
               : conv_typed<__nv_bfloat16>(x, x_pitch, cp, taps, w, bias, state, tk, out, carry, st);
}

jsm_status scan_conv_launch(bool f32, const ScanDims& d, const ScanWeights& w, const ScanState& s, const StepTokens& tk, const void* xz,
                            void* xc, bool carry, cudaStream_t st) {
    return short_conv_launch(f32, xz, 2 * d.ip(), d.ip(), d.taps, w.conv, w.conv_b, s.conv, tk, xc, carry, st);
}

template <typename T>
__global__ void __launch_bounds__(256) conv_carry_kernel(const T* __restrict__ x, long long pitch, T* state, const int32_t* __restrict__ seg_start,
                                                         const int32_t* __restrict__ seg_len, const int32_t* __restrict__ seg_pos0,
                                                         const int32_t* __restrict__ seg_slot, int cp, int taps) {
    chain_trigger();
    chain_wait();
    const int c = blockIdx.x * 256 + threadIdx.x, seg = blockIdx.y;
    if (c < cp) carry_conv_state(state + (long long)seg_slot[seg] * (taps - 1) * cp, x, pitch, c, cp, taps, seg_start[seg], seg_len[seg], seg_pos0[seg]);
}
jsm_status short_conv_carry_launch(bool f32, const void* x, long long x_pitch, int cp, int taps, void* state, const StepTokens& tk, cudaStream_t st) {
    if (taps <= 1) return JSM_OK;
    const dim3 grid((cp + 255) / 256, tk.n_segs);
    if (f32) JSM_CUDA_CHECK(launch_chained(conv_carry_kernel<float>, grid, dim3(256), 0, st, (const float*)x, x_pitch, (float*)state, tk.seg_start, tk.seg_len,
                                           tk.seg_pos0, tk.seg_slot, cp, taps));
    else JSM_CUDA_CHECK(launch_chained(conv_carry_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, (const __nv_bfloat16*)x, x_pitch, (__nv_bfloat16*)state,
                                       tk.seg_start, tk.seg_len, tk.seg_pos0, tk.seg_slot, cp, taps));
    JSM_LAUNCH_CHECK();
    return JSM_OK;
}

static ScanArgs scan_args(const ScanDims& d, const ScanWeights& w, const ScanState& s, const StepTokens& tk, const void* xz, const void* xc,
                          const float* proj, const float* dt_raw, void* y) {
    ScanArgs a;
    a.A = w.A; a.D = w.D; a.dt_b = w.dt_b; a.proj = proj; a.dt_raw = dt_raw; a.xz = xz; a.xc = xc; a.dt_w = w.dt; a.y = y;
    a.conv = s.conv; a.S = s.S;
    a.seg_start = tk.seg_start; a.seg_len = tk.seg_len; a.seg_pos0 = tk.seg_pos0; a.seg_slot = tk.seg_slot;
    a.ip = d.ip(); a.np = d.np(); a.rp = d.rp(); a.state = d.state; a.taps = d.taps; a.n_segs = tk.n_segs;
    return a;
}

template <typename T, int NS>
static jsm_status scan_go(const ScanArgs& a, cudaStream_t st) {
    constexpr int smem = scan_smem<T, NS>();
    static DeviceOnce once;  // per instantiation
    JSM_CUDA_CHECK(allow_shared(once, scan_kernel<T, NS>, smem));
    JSM_CUDA_CHECK(launch_spread(scan_kernel<T, NS>, dim3((a.ip + SC_CH - 1) / SC_CH, a.n_segs), dim3(SC_THREADS), smem, st, a));
    JSM_LAUNCH_CHECK();
    return JSM_OK;
}
template <typename T, int NP>
static jsm_status step_go(const ScanArgs& a, cudaStream_t st) {
    const size_t smem = (size_t)ST_BB * (2 * a.np + (sizeof(T) == 2 ? 0 : a.rp)) * sizeof(float);
    static DeviceOnce once;  // per instantiation
    JSM_CUDA_CHECK(allow_shared(once, scan_step_kernel<T, NP>, 200 * 1024));
    JSM_CUDA_CHECK(launch_chained(scan_step_kernel<T, NP>, dim3((a.ip + ST_CH - 1) / ST_CH, (a.n_segs + ST_BB - 1) / ST_BB), dim3(ST_THREADS), smem, st, a));
    JSM_LAUNCH_CHECK();
    return JSM_OK;
}
static jsm_status scan_wide_go(const ScanArgs& a, cudaStream_t st) {
    static DeviceOnce once;
    JSM_CUDA_CHECK(allow_shared(once, scan_wide_kernel, (int)sizeof(ScanWideShared)));
    JSM_CUDA_CHECK(launch_spread(scan_wide_kernel, dim3((a.ip + SW_CH - 1) / SW_CH, a.n_segs), dim3(SW_THREADS), sizeof(ScanWideShared), st, a));
    JSM_LAUNCH_CHECK();
    return JSM_OK;
}
// the smallest instance whose threads hold a channel's states
template <typename T>
static jsm_status scan_dispatch(const ScanArgs& a, cudaStream_t st) {
    // Two blocks of scan_kernel fit beside one another on an SM without slowing each other down much (2048 tokens, scan_kernel / scan_wide_kernel, us with
    // cold caches: 128 blocks 109 / 132, 256 blocks 131 / 134, 296 blocks 132 / 134, 300 blocks 158 / 135, 384 blocks 160 / 137, 512 blocks 194 / 139; 300
    // tokens: 296 blocks 24.5 / 25.3, 304 blocks 28.2 / 25.1; 64 tokens: 296 blocks 9.3 / 9.8, 304 blocks 10.3 / 10.2, 512 blocks 11.9 / 10.4).
    if constexpr (sizeof(T) == 2)
        if (a.state > 8 && a.state <= 16 && (long long)((a.ip + SC_CH - 1) / SC_CH) * a.n_segs > 2ll * sm_count()) return scan_wide_go(a, st);
    return a.state <= 8 ? scan_go<T, 1>(a, st) : a.state <= 16 ? scan_go<T, 2>(a, st) : a.state <= 24 ? scan_go<T, 3>(a, st)
         : a.state <= 32 ? scan_go<T, 4>(a, st) : a.state <= 64 ? scan_go<T, 8>(a, st) : scan_go<T, 16>(a, st);
}
template <typename T>
static jsm_status step_dispatch(const ScanArgs& a, cudaStream_t st) {
    return a.np <= 8 ? step_go<T, 2>(a, st) : a.np <= 16 ? step_go<T, 4>(a, st) : a.np <= 32 ? step_go<T, 8>(a, st) : step_go<T, 0>(a, st);
}

jsm_status scan_launch(bool f32, const ScanDims& d, const ScanWeights& w, const ScanState& s, const StepTokens& tk, const void* xz,
                       const void* xc, const float* proj, const float* dt_raw, void* y, cudaStream_t st) {
    if (d.state > 128) JSM_FAIL(JSM_UNSUPPORTED, "selective scan: %d states per channel (at most 128)", d.state);
    const ScanArgs a = scan_args(d, w, s, tk, xz, xc, proj, dt_raw, y);
    return f32 ? scan_dispatch<float>(a, st) : scan_dispatch<__nv_bfloat16>(a, st);
}

jsm_status scan_step_launch(bool f32, const ScanDims& d, const ScanWeights& w, const ScanState& s, const StepTokens& tk, const void* xz,
                            const void* xc, const float* proj, void* y, cudaStream_t st) {
    if (d.state > 128) JSM_FAIL(JSM_UNSUPPORTED, "selective scan: %d states per channel (at most 128)", d.state);
    const ScanArgs a = scan_args(d, w, s, tk, xz, xc, proj, nullptr, y);
    return f32 ? step_dispatch<float>(a, st) : step_dispatch<__nv_bfloat16>(a, st);
}

jsm_status scan_dt_operand_launch(const ScanDims& d, const float* proj, void* out, int T, cudaStream_t st) {
    const long long n = (long long)T * (d.rp() / 8);
    JSM_CUDA_CHECK(launch_chained(scan_dt_operand_kernel, dim3((unsigned)std::min<long long>((n + 255) / 256, 148 * 8)), dim3(256), 0, st, proj,
                                  (__nv_bfloat16*)out, T, d.rp(), d.proj_cols()));
    JSM_LAUNCH_CHECK();
    return JSM_OK;
}

}  // namespace jsm
