// bf16 projections of a few dozen tokens (17 to 128; fewer where a matrix has few tiles) over packed weights (the layout of linear_packed.cu): Y[t, n] = sum_k X[t, k] W[n, k],
// the batched decode step's and short prompt's form of weight_net_t::forward (mat_net_t.hpp:38-49).
//
// What bounds it.  The weights are read once, so the floor is the memory's; but a launch moves only 8 to 50 MB (1.3 to 8 us), and
// what surrounds the stream decides: how many multiprocessors take part, and the tail between the last product and the last
// store.  The streaming kernel formed clusters of eight CTAs for narrow matrices, of which the chip holds 15 and got 16: a second wave
// of clusters started when the first had ended.  64 tokens, back to back, there -> here: 2048 x 2048 f32 out 12.4 -> 6.5 us,
// 2048 x 5504 17.6 -> 9.9, 6144 x 2048 10.2 -> 9.6, gate/up 5504 x 2048 14.5 -> 13.8, 4096 x 4096 10.8 -> 10.3, 4096 x 11008 20.8 -> 20.4.
// Time stamps: 0.5 to 2 us from the predecessor's end to the first products, 1.1 us from the accumulator to the folded sums, 0.7 to
// 1.5 us of epilogue.  The loops of drain and epilogue are rolled: unrolled they took 0.7 us more each (code fetched cold).
//
// Split.  A cluster of S CTAs takes one tile of 128 packed rows (or, for narrow matrices, half of one: 64 rows) x all tokens,
// an S-th of the depth each; S and the height come from a cost estimate over what the chip holds at once (mid_shape).
//
// Fold.  The tokens of the tile belong to the cluster's CTAs in equal shares.  Every CTA writes its fp32 partial sums straight from
// tensor memory into the owners' shared memory (a warp stores 128 contiguous bytes per token) and signals their barriers; an
// owner waits for its own barrier only, adds in rank order and runs the epilogue.  One one-way trip: no barrier before the reads,
// no remote reads, none after them.
//
// Roles (384 threads): warp 0 streams weights, warp 2 tokens, warp 1 issues the products, warps 4-11 drain and finish (two per
// quadrant of TMEM lanes, half of the tokens each).
#include "tc_utils.cuh"
#include "linear_bf16.cuh"
#include "linear_epilogue.cuh"
#include <algorithm>
#include <mutex>

namespace jsm {

using namespace tc;

constexpr int LM_THREADS = 384, LM_EPI = 8;
constexpr uint32_t LM_UNIT = 128 * 64 * 2;  // a packed unit: 128 rows x 64 k

struct LmParams {
    int T, N, kbt;
    int half;                // tiles of 64 packed rows
    int epilogue, out_f32;
    const uint8_t* Wp;
    const float* bias;
    const __nv_bfloat16* R;
    void* Y;
    const float* ssq_in;
    int ssq_in_tiles, ssq_stride;
    float inv_d, eps;
    float* ssq_out;
    float glu_alpha, glu_limit;
    int* err;
    unsigned long long* trace;
    int trace_ctas;
};

__device__ __forceinline__ uint32_t lm_reg_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t lm_reg_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void lm_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void lm_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t lm_peer(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void lm_store_peer(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void lm_arrive_peer(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait for arrivals of other CTAs (acquires at cluster scope)
__device__ __forceinline__ bool lm_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err, int code) {
    const long long t0 = clock64();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
            *abort_flag = 1;
            if (err) atomicCAS(err, 0, code);
            return false;
        }
    }
}

// KIND: 0 plain (optionally a fused norm's row factor, row statistics), 1 the same with bias and activations, 2 gate/up pairs, 3 with a residual
constexpr int lm_stages(int bn) { return bn <= 32 ? 4 : bn == 64 ? 3 : 2; }
constexpr int lm_smem(int bn) { return lm_stages(bn) * 2 * ((int)LM_UNIT + bn * 128) + (bn + 64) * 512 + 1024; }

// TRACED: an image of its own for launches that record time stamps (tests of a null pointer in every launch cost 0.1 us)
#define LM_STAMP(slot) do { if constexpr (TRACED) lin_stamp(P.trace, P.trace_ctas, slot); } while (0)
template <int BN, int KIND, bool TRACED>
__global__ void __launch_bounds__(LM_THREADS, 1) linear_mid_kernel(const __grid_constant__ CUtensorMap tmap_x, LmParams P) {
    constexpr int STAGES = lm_stages(BN);
    constexpr uint32_t X_BYTES = BN * 128, X_OFF = 2 * LM_UNIT, STAGE = 2 * (LM_UNIT + X_BYTES);
    constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
    constexpr bool PAIRED = KIND == 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* red = reinterpret_cast<float*>(tiles + STAGES * STAGE);  // [rank][own token][128]
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full, red_full;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;
    __shared__ float row_scale[BN];

    chain_trigger();
    if (threadIdx.x == 0) LM_STAMP(0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)lm_reg_size(), rank = (int)lm_reg_rank(), tile = (int)blockIdx.x / S;
    const int kb0 = P.kbt * rank / S, kb1 = P.kbt * (rank + 1) / S;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 2);  // the weights' and the tokens' producer
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_full, 1);
        mbar_init(&red_full, LM_EPI * S);
        mbar_fence_init();
        tma_prefetch_desc(&tmap_x);
    }
    if (warp == 1) {
        tmem_alloc(&tmem_base_smem, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    lm_cluster_arrive();  // this CTA's barriers exist; waited for before the first remote store
    const uint32_t tmem = tmem_base_smem;

    if (warp == 0) {
        const int rows = P.half ? 64 : 128;
        const uint8_t* src = P.Wp + (size_t)(P.half ? tile >> 1 : tile) * P.kbt * LM_UNIT + (P.half ? (tile & 1) * 8192 : 0);
        int s = 0, n_issued = 0;
        uint32_t ph = 0;
        for (int kb = kb0; kb < kb1; kb += 2, ++n_issued) {
            if (n_issued >= STAGES && !mbar_wait_warp(&empty_bar[s], ph ^ 1, &abort_flag, P.err, TC_TIMEOUT_EMPTY)) break;
            const int n = min(2, kb1 - kb);
            if (elect_one()) {
                mbar_expect_tx(&full_bar[s], (uint32_t)(n * rows * 128));
                if (P.half)
                    for (int q = 0; q < n; ++q) bulk_load(tiles + s * STAGE + q * LM_UNIT, src + (size_t)(kb + q) * LM_UNIT, 8192, &full_bar[s]);
                else bulk_load(tiles + s * STAGE, src + (size_t)kb * LM_UNIT, (uint32_t)n * LM_UNIT, &full_bar[s]);
            }
            __syncwarp();
            if (n_issued == STAGES - 1 && lane == 0) LM_STAMP(1);
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (abort_flag) {  // let the copies in flight land (bounded)
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
        lm_cluster_wait();
        lm_cluster_arrive();
    } else if (warp == 2) {
        chain_wait();
        if (lane == 0) LM_STAMP(2);
        int s = 0, i = 0;
        uint32_t ph = 0;
        for (int kb = kb0; kb < kb1; kb += 2, ++i) {
            if (i >= STAGES && !mbar_wait_warp(&empty_bar[s], ph ^ 1, &abort_flag, P.err, TC_TIMEOUT_EMPTY)) break;
            const int n = min(2, kb1 - kb);
            if (elect_one()) {
                mbar_expect_tx(&full_bar[s], (uint32_t)n * X_BYTES);
                for (int q = 0; q < n; ++q) tma_load_2d(tiles + s * STAGE + X_OFF + q * X_BYTES, &tmap_x, (kb + q) * 64, 0, &full_bar[s]);
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (abort_flag) {
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
        lm_cluster_wait();
        lm_cluster_arrive();
    } else if (warp == 1) {
        constexpr uint32_t idesc = instr_desc_bf16(128, BN);  // (of a half tile the upper 64 rows multiply what is there and nobody reads them)
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int kb = kb0; kb < kb1; kb += 2) {
            ok = mbar_wait_warp(&full_bar[s], ph, &abort_flag, P.err, TC_TIMEOUT_FULL);
            if (!ok) break;
            if (kb == kb0 && lane == 0) LM_STAMP(3);
            tc_fence_after();
            const uint32_t addr = smem_u32(tiles + s * STAGE);
            const bool both = kb + 1 < kb1;
            if (elect_one()) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (q == 0 || both) {
                        const uint64_t a = smem_desc_sw128(addr + q * LM_UNIT), b = smem_desc_sw128(addr + X_OFF + q * X_BYTES);
#pragma unroll
                        for (int k = 0; k < 4; ++k) mma_ss(tmem, a + (uint64_t)(k * 2), b + (uint64_t)(k * 2), idesc, (kb > kb0 || q > 0 || k > 0) ? 1u : 0u);
                    }
                mma_commit(&empty_bar[s]);
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok && elect_one()) mma_commit(&acc_full);
        __syncwarp();
        if (lane == 0) LM_STAMP(4);
        lm_cluster_wait();
        lm_cluster_arrive();
    } else if (warp >= 4) {
        const int quad = warp & 3, part = (warp - 4) >> 2, row = quad * 32 + lane, etid = threadIdx.x - 128;
        const int share = ((P.T + S - 1) / S + 7) & ~7, t_lo = min(P.T, rank * share), n_own = min(share, P.T - t_lo);  // (tokens in eights: a load from tensor memory has one owner)
        constexpr int ITEMS = BN / 8;  // pieces of four features per thread: up to BN tokens x 32 pieces / 256 threads
        const int shift = PAIRED || P.half ? 4 : 5, mask = (1 << shift) - 1;
        const int n_tile0 = PAIRED || P.half ? tile * 64 : tile * 128;
        const int f4 = (etid & mask) * 4, n = n_tile0 + f4;
        const bool n_ok = n < P.N;
        chain_wait();
        if (P.ssq_in) {  // factor of a fused RMSNorm: the per-tile sums of squares of the token's row, added in tile order
            for (int t = etid; t < n_own; t += 32 * LM_EPI) {
                float q = 0.0f;
                int j = 0;
                for (; j + 8 <= P.ssq_in_tiles; j += 8) {
                    float v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = __ldcg(P.ssq_in + (size_t)(j + k) * P.ssq_stride + t_lo + t);
#pragma unroll
                    for (int k = 0; k < 8; ++k) q += v[k];
                }
                for (; j < P.ssq_in_tiles; ++j) q += __ldcg(P.ssq_in + (size_t)j * P.ssq_stride + t_lo + t);
                row_scale[t] = rsqrtf(q * P.inv_d + P.eps);
            }
        }
        uint2 rr[KIND == 3 ? ITEMS : 1];  // the residual is requested while the weights stream
        if constexpr (KIND == 3)
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const int lt = (i * 256 + etid) >> shift;
                rr[i] = lt < n_own && n_ok ? *reinterpret_cast<const uint2*>(P.R + (size_t)(t_lo + lt) * P.N + n) : make_uint2(0u, 0u);
            }
        const float4 bias = (KIND == 1 || KIND == 3) && P.bias && n_ok ? *reinterpret_cast<const float4*>(P.bias + n) : make_float4(0.f, 0.f, 0.f, 0.f);
        lm_cluster_wait();  // the peers' barriers exist
        const bool acc_ok = mbar_wait(&acc_full, 0, &abort_flag, P.err, TC_TIMEOUT_ACC);
        tc_fence_after();
        const uint32_t red_addr = smem_u32(red) + row * 4;
        if (acc_ok && !(P.half && quad >= 2) && part * (BN / 2) < P.T) {
            const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16) + part * (BN / 2);
#pragma unroll 1
            for (int c = 0; c < BN / 2; c += 8) {  // (short code: it is fetched once per launch, cold)
                const int t = part * (BN / 2) + c, owner = t / share;
                if (t >= P.T) break;
                uint32_t r[8];
                tmem_ld8(acc + c, r);
                const uint32_t dst = lm_peer(red_addr + (rank * share + t - owner * share) * 512, owner);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) lm_store_peer(dst + j * 512, r[j]);
            }
        }
        tc_fence_before();
        __syncwarp();
        if (S == 1) {
            if (lane == 0) mbar_arrive(&red_full);
        } else if (lane < S) lm_arrive_peer(lm_peer(smem_u32(&red_full), lane));
        asm volatile("bar.sync 1, 256;" ::: "memory");  // row_scale
        const bool ok = lm_wait_cluster(&red_full, 0, &abort_flag, P.err, TC_TIMEOUT_MISC) && acc_ok;
        lm_cluster_arrive();  // nothing of the peers is written or awaited any more
        if (ok) {
            auto sum = [&](int lt, int at) {
                float4 v = *reinterpret_cast<const float4*>(red + lt * 128 + at);
                for (int z = 1; z < S; ++z) {
                    const float4 w = *reinterpret_cast<const float4*>(red + (z * share + lt) * 128 + at);
                    v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
                }
                return v;
            };
            auto finish = [&](int lt, const uint2& res) {
                const int t = t_lo + lt;
                const float sc = P.ssq_in ? row_scale[lt] : 1.0f;
                float4 v = sum(lt, f4);
                v.x *= sc; v.y *= sc; v.z *= sc; v.w *= sc;
                if constexpr (PAIRED) {
                    float4 u = sum(lt, f4 + 64);
                    u.x *= sc; u.y *= sc; u.z *= sc; u.w *= sc;
                    if (P.epilogue == LIN_CLAMPED_GLU) {
                        v.x = pk_clamped_glu(v.x, u.x, P.glu_alpha, P.glu_limit); v.y = pk_clamped_glu(v.y, u.y, P.glu_alpha, P.glu_limit);
                        v.z = pk_clamped_glu(v.z, u.z, P.glu_alpha, P.glu_limit); v.w = pk_clamped_glu(v.w, u.w, P.glu_alpha, P.glu_limit);
                    } else if (P.epilogue == LIN_GELU_GLU) {
                        v.x = pk_gelu_glu(v.x, u.x); v.y = pk_gelu_glu(v.y, u.y); v.z = pk_gelu_glu(v.z, u.z); v.w = pk_gelu_glu(v.w, u.w);
                    } else {
                        v.x = pk_silu(v.x) * u.x; v.y = pk_silu(v.y) * u.y; v.z = pk_silu(v.z) * u.z; v.w = pk_silu(v.w) * u.w;
                    }
                } else {
                    if constexpr (KIND == 1 || KIND == 3) {
                        v.x += bias.x; v.y += bias.y; v.z += bias.z; v.w += bias.w;
                        if (KIND == 1 && P.epilogue == LIN_RELU) {
                            v.x = fmaxf(v.x, 0.0f); v.y = fmaxf(v.y, 0.0f); v.z = fmaxf(v.z, 0.0f); v.w = fmaxf(v.w, 0.0f);
                        } else if (KIND == 1 && P.epilogue == LIN_GELU) {
                            v.x = pk_gelu(v.x); v.y = pk_gelu(v.y); v.z = pk_gelu(v.z); v.w = pk_gelu(v.w);
                        }
                    }
                    if constexpr (KIND == 3) {
                        v.x += bf16lo(res.x); v.y += bf16hi(res.x); v.z += bf16lo(res.y); v.w += bf16hi(res.y);
                    }
                }
                if (P.out_f32) {
                    if (n_ok) *reinterpret_cast<float4*>(static_cast<float*>(P.Y) + (size_t)t * P.N + n) = v;
                } else {
                    const uint2 o = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
                    if (n_ok) *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(P.Y) + (size_t)t * P.N + n) = o;
                    if (!PAIRED && P.ssq_out) {  // (full tiles: a warp has one token)
                        const float a = bf16lo(o.x), b = bf16hi(o.x), c = bf16lo(o.y), e = bf16hi(o.y);
                        const float q = warp_sum(n_ok ? (a * a + b * b) + (c * c + e * e) : 0.0f);
                        if (lane == 0) P.ssq_out[(size_t)tile * P.ssq_stride + t] = q;
                    }
                }
            };
            if constexpr (PAIRED) {
#pragma unroll 1
                for (int lt = etid >> shift; lt < n_own; lt += 256 >> shift)
                    if (n_ok) finish(lt, make_uint2(0u, 0u));
            } else if (KIND == 3) {
#pragma unroll
                for (int i = 0; i < (KIND == 3 ? ITEMS : 0); ++i) {
                    const int lt = (i * 256 + etid) >> shift;
                    if (lt < n_own) finish(lt, rr[i]);
                }
            } else {
#pragma unroll 1
                for (int lt = etid >> shift; lt < n_own; lt += 256 >> shift) finish(lt, make_uint2(0u, 0u));
            }
        }
        if (etid == 0) LM_STAMP(5);
    } else {
        lm_cluster_wait();
        lm_cluster_arrive();
    }
    tc_fence_before();
    __syncwarp();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
    lm_cluster_wait();  // no CTA leaves while a peer may still write into it
    if (threadIdx.x == 0) LM_STAMP(7);
}

// clusters of S CTAs that the chip holds at once (15 of eight, 33 of four, 45 of three, although it has 148 multiprocessors)
template <int BN, int KIND, bool TRACED>
static int mid_capacity(int S) {
    static std::mutex mu;
    static int known[64][9];  // per device
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return S == 1 ? sm_count() : sm_count() / S * 3 / 4;
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev][S] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(S * 256);
        cfg.blockDim = dim3(LM_THREADS);
        cfg.dynamicSmemBytes = lm_smem(BN);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = S;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, linear_mid_kernel<BN, KIND, TRACED>, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = S == 1 ? sm_count() : sm_count() / S * 3 / 4;
        }
        known[dev][S] = n;
    }
    return known[dev][S];
}

// CTAs per tile and the tile's height.  A CTA takes 0.3 us per unit of 64 k of a whole tile (the rate of one multiprocessor's copies; beyond 64
// tokens their bytes show: 0.36), or its share of the memory's 6.4 TB/s, and about 4 us around it; clusters that do not fit at once
// wait for the first ones.  A unit of a half tile brings the same bytes of tokens: 0.17 us up to 16 of them, 0.19 up to 32, 0.24 up to 64, 0.355
// up to 128.  8192 x 4096 over 32, 64 and 100 tokens: 128 half tiles 15.1, 18.2 and 27.0 us, 64 clusters of two 12.9, 14.3 and 18.4 us;
// 2048 x 1024 over 64: half tiles 4.9 us, whole ones 5.4.
template <int BN, int KIND, bool TRACED>
static void mid_shape(int n_tiles, int kbt, bool may_halve, int* S_out, int* half_out) {
    constexpr float whole_us = BN <= 64 ? 0.3f : 0.36f, half_us = BN == 16 ? 0.17f : BN == 32 ? 0.19f : BN == 64 ? 0.24f : 0.355f;
    constexpr float half_around = BN == 16 ? 4.0f : 3.5f;
    float best = 0.0f;
    *S_out = 0;
    for (int half = 0; half <= (may_halve ? 1 : 0); ++half)
        for (int S = 1; S <= 8 && S <= kbt; ++S) {
            const int tiles = n_tiles << half, cap = mid_capacity<BN, KIND, TRACED>(S), at_once = std::min(tiles, cap) * S;
            const float unit = std::max(half ? half_us : whole_us, (half ? 0.5f : 1.0f) * 16.384e-3f * (float)at_once / 6.4f);
            const float cost = (float)((tiles + cap - 1) / cap) * ((half ? half_around : 4.0f) + (S > 1 ? 0.5f : 0.0f) + (float)((kbt + S - 1) / S) * unit);
            if (*S_out == 0 || cost < best) { best = cost; *S_out = S; *half_out = half; }
        }
}

template <int BN, int KIND, bool TRACED = false>
static jsm_status launch_mid(const PackedArgs& a, LmParams& P, int n_tiles, cudaStream_t st) {
    if (!TRACED && (P.trace = linear_trace_next(&P.trace_ctas))) return launch_mid<BN, KIND, true>(a, P, n_tiles, st);
    static DeviceOnce once;  // per instantiation
    JSM_CUDA_CHECK(allow_shared(once, linear_mid_kernel<BN, KIND, TRACED>, lm_smem(BN)));
    int S, half;
    mid_shape<BN, KIND, TRACED>(n_tiles, P.kbt, KIND != 2 && !a.ssq_out, &S, &half);
    P.half = half;
    CUtensorMap mx;
    jsm_status s = make_tmap_bf16_2d(&mx, a.X, (uint64_t)a.T, (uint64_t)a.K, (uint64_t)(a.x_row_stride > 0 ? a.x_row_stride : a.K), BN, 64);
    if (s != JSM_OK) return s;
    const int tiles = half ? (a.N + 63) / 64 : n_tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * S);
    cfg.blockDim = dim3(LM_THREADS);
    cfg.dynamicSmemBytes = lm_smem(BN);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.chained && chained_launch_enabled() ? 2 : 1;
    JSM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, linear_mid_kernel<BN, KIND, TRACED>, mx, P));
    g_launches.fetch_add(1);
    return JSM_OK;
}

// Arguments checked by linear_packed_tokens.
jsm_status linear_mid_launch(const PackedArgs& a, cudaStream_t st) {
    const int paired = a.epilogue == LIN_SILU_MUL || a.epilogue == LIN_CLAMPED_GLU || a.epilogue == LIN_GELU_GLU;
    LmParams P;
    int n_tiles;
    pk_dims(a.N, a.K, paired, &n_tiles, &P.kbt);
    P.T = a.T; P.N = a.N; P.half = 0;
    P.epilogue = a.epilogue; P.out_f32 = a.out_f32 ? 1 : 0;
    P.Wp = static_cast<const uint8_t*>(a.Wp);
    P.bias = a.bias; P.R = static_cast<const __nv_bfloat16*>(a.R); P.Y = a.Y;
    P.ssq_in = a.ssq_in; P.ssq_in_tiles = a.ssq_in_tiles; P.ssq_stride = a.ssq_stride > 0 ? a.ssq_stride : a.T;
    P.inv_d = 1.0f / (float)a.K; P.eps = a.eps; P.ssq_out = a.ssq_out;
    P.glu_alpha = a.glu_alpha; P.glu_limit = a.glu_limit;
    P.err = tc_error_word();
    const int kind = paired ? 2 : a.epilogue == LIN_RESIDUAL ? 3 : a.bias || a.epilogue == LIN_RELU || a.epilogue == LIN_GELU ? 1 : 0;
#define LM_GO(BN_) \
    return kind == 3 ? launch_mid<BN_, 3>(a, P, n_tiles, st) : kind == 2 ? launch_mid<BN_, 2>(a, P, n_tiles, st) \
         : kind == 1 ? launch_mid<BN_, 1>(a, P, n_tiles, st) : launch_mid<BN_, 0>(a, P, n_tiles, st)
    if (a.T <= 16) LM_GO(16);
    if (a.T <= 32) LM_GO(32);
    if (a.T <= 64) LM_GO(64);
    LM_GO(128);
#undef LM_GO
}

}  // namespace jsm
