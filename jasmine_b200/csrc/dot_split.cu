// fp32 products of many tokens on the tensor cores: C[t, n] = sum_k X[t, k] W[n, k] with fp32 operands, sums and results, the prompts' form of
// weight_net_t::forward (mat_net_t.hpp:38-49) in f32 models.
//
// Method.  An fp32 number is the sum of three bf16 numbers, x = h + m + l, each the rest of the one before rounded to 8 bits: 24 bits,
// nothing is lost (splitting fp32 into bf16 numbers for matrix units: Henry, Tang, Heinecke, "Leveraging the bfloat16 artificial intelligence
// datatype for higher-precision computations", 2019).  Of the nine products of two such sums the six largest are taken, the smallest first; of the others m l
// and l m are 2^-25 of the product each at most, l l 2^-34.  The tensor core truncates: an addition to a running sum drops what lies below its
// last place, always toward zero.  So no large product is ever added to another one there except within one MMA of 16: a block of
// 64 products has four accumulators, one per step, the first of which also takes all the small products before its large ones; they are added in
// registers, rounded to nearest, and the ranks of a cluster with what each rounding leaves out.  A block of weights whose m or l parts are all zero
// (weights that came as bf16) leaves those products out: the sums are the same to the bit.
//
// Error against 64 bits, rms, fp32 chains -> here: operands of random sign 0.83e-7 -> 0.49e-7 (64 products), 1.05e-7 -> 0.61e-7 (1024), 1.17e-7 ->
// 0.72e-7 (2752); of one sign 0.48e-7 -> 0.45e-7, 0.52e-7 -> 0.39e-7, 0.49e-7 -> 0.34e-7 (one accumulator per block: 0.95e-7, two: 0.65e-7),
// and where a CTA adds all blocks of 1024 products by itself 0.64e-7 -> 0.67e-7 (random signs: 1.16e-7 -> 0.89e-7).
//
// What bounds it.  The fp32 pipe ran at half of its rate at best; 300 tokens, there -> here, us: 1024 x 1024 41 -> 13, 1024 x 2752 59 -> 24, 2752 x 1024
// 53 -> 22, 8000 x 1024 151 -> 63 (weights that fit bf16: 12, 22, 20, 56); 33 tokens: 1024 x 2752 26 -> 14; 1 token: 8000 x 1024 22 -> 15.
// A block of products takes 12 to 24 MMAs, and taking the operands apart is the longer part: about 70 instructions per eight numbers,
// half of the issue slots, and the latency of the next block's loads behind them (1.0 to 1.6 us a block; twice the warps, or the
// weights' lines asked into L2 four blocks ahead: 5 to 30 % slower).  So few CTAs share an operand's rows as possible: 128 features and up to
// 128 tokens per CTA, and a cluster of CTAs shares the products of a tile.  The four accumulators cost 3 to 11 % (300 x 2752 x 1024 in pairs
// 29.7 -> 32.8): they fill the tensor memory, so a block's MMAs wait until the block before it has been added, which the splitting hides.
//
// Roles (512 threads, a whole number of warps per scheduler: 128 registers each): warps 0-7 read fp32 rows, take them apart and write the
// three planes of a block into shared memory (128-byte swizzle, two stages); warps 8-15 add the blocks' sums (two per quadrant of TMEM
// lanes, half of the tokens each); warp 8 also issues the MMAs (features are the rows, tokens the columns).
//
// Gate and up projections of a feed-forward run as pairs: 64 features' gate and up rows make one tile, and the activation follows where the sums meet (the
// two products and a launch for the activation, 300 x 2752 x 1024: 43 us, here 33; 38 with weights of 24 bits).
//
// Range.  Both operands are scaled by 2^39 on the way in, so that every fp32 number, the subnormal ones too, keeps all its parts, and the sums by 2^-78 on the
// way out.  What leaves the range then (infinities, NaN, operands above 2^88, sums above 2^49) comes out as no finite number, and every such result is
// formed again by plain fp32 additions.
#include "tc_utils.cuh"
#include "linear_epilogue.cuh"
#include "mma_utils.cuh"
#include <algorithm>
#include <mutex>

namespace jsm {

using namespace tc;

constexpr int DS_SPLIT_WARPS = 8, DS_ADD_WARPS = 8, DS_THREADS = 32 * (DS_SPLIT_WARPS + DS_ADD_WARPS);
constexpr int DS_KB = 64, DS_ROWS = 128;
constexpr int ds_plane(int bn) { return (DS_ROWS + bn) * 128; }
constexpr int ds_smem(int bn) { return 2 * 3 * ds_plane(bn) + 1024; }

struct DotSplitParams {
    const float *X, *W, *W2;  // W2: the up rows of gate / up pairs
    float* C;
    long long ldx, ldw, ldc;
    int T, N, K, tok_blocks;
    int* err;
    int gelu;                 // pairs: the activation, and what the clamped one needs
    float alpha, limit;
};

__device__ __forceinline__ uint32_t ds_cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t ds_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ds_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// two numbers -> the next bf16 part of each; what is left stays in a and b
__device__ __forceinline__ uint32_t ds_part(float& a, float& b) {
    const uint32_t p = pack_bf16x2(a, b);
    a -= bf16lo(p);
    b -= bf16hi(p);
    return p;
}

// Operands are scaled on the way in: the smallest number that fp32 holds, 2^-149, keeps its parts above 2^-133, where bf16 ends
constexpr float DS_SCALE = 0x1p39f, DS_BACK = 1.0f / (DS_SCALE * DS_SCALE);

// sum += q; what the rounding leaves out goes to lost
__device__ __forceinline__ void ds_add(float& sum, float& lost, float q) {
    const float t = sum + q, p = t - sum;
    lost += (sum - (t - p)) + (q - p);
    sum = t;
}
// Products of one row of X with four rows of W by plain fp32 additions: blocks of 32 in two chains, as dot_f32_kernel adds them (what overflows on the
// way is the same).  rows: bit j, whether number j is formed again.
static __device__ __noinline__ float4 ds_again(float4 old, uint32_t rows, const float* w, long long ldw, const float* x, int K) {
    float v[4] = {old.x, old.y, old.z, old.w};
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        if (!(rows >> j & 1)) continue;
        float sum = 0.0f, lost = 0.0f;
        for (int k0 = 0; k0 < K && sum == sum; k0 += 32) {
            float even = 0.0f, odd = 0.0f;
#pragma unroll
            for (int k = k0; k < k0 + 32; k += 4) {
                if (k >= K) break;
                const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + j * ldw + k);
                even = fmaf(a.x, b.x, even); odd = fmaf(a.y, b.y, odd);
                even = fmaf(a.z, b.z, even); odd = fmaf(a.w, b.w, odd);
            }
            ds_add(sum, lost, even + odd);
        }
        if (fabsf(sum + lost) < INFINITY) sum += lost;
        if (j == 0) v[0] = sum;
        else if (j == 1) v[1] = sum;
        else if (j == 2) v[2] = sum;
        else v[3] = sum;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// BN: tokens of a tile.  PAIRED: a tile has the gate rows of 64 features, then their up rows; C = activation(gate, up)
template <int BN, bool PAIRED>
__global__ void __launch_bounds__(DS_THREADS, 1) dot_split_kernel(DotSplitParams P) {
    constexpr int FEATURES = PAIRED ? DS_ROWS / 2 : DS_ROWS;
    constexpr int PLANE = ds_plane(BN), STAGE = 3 * PLANE, X_OFF = DS_ROWS * 128;
    constexpr int ROWS_PASS = DS_SPLIT_WARPS * 4, W_ITEMS = DS_ROWS / ROWS_PASS, X_ITEMS = BN / ROWS_PASS, ITEMS = W_ITEMS + X_ITEMS;
    constexpr uint32_t BUF = BN <= 32 ? 32 : BN <= 64 ? 64 : 128;  // tensor-memory columns between the four accumulators
    constexpr int COLS = BN / 2;                                   // columns of an adding warp
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[2], empty_bar[2], acc_full, acc_empty;
    __shared__ uint32_t w_parts[2][DS_SPLIT_WARPS];  // which of a block's weights have an m part (1), an l part (2)
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;

    chain_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)ds_cluster_size(), rank = (int)ds_cluster_rank(), tile = (int)blockIdx.x / S;
    const int n0 = tile / P.tok_blocks * FEATURES, t0 = tile % P.tok_blocks * BN;
    const int blocks = (P.K + DS_KB - 1) / DS_KB, b0 = blocks * rank / S, b1 = blocks * (rank + 1) / S;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full_bar[s], DS_SPLIT_WARPS);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_full, 1);
        mbar_init(&acc_empty, DS_ADD_WARPS);
        mbar_fence_init();
    }
    if (warp == DS_SPLIT_WARPS) {
        tmem_alloc(&tmem_base_smem, 4 * BUF);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_smem;
    float acc[COLS];

    if (warp < DS_SPLIT_WARPS) {
        // eight lanes take a row's 64 numbers; a pass of the eight warps covers 32 rows
        const int r0 = warp * 4 + (lane >> 3), chunk = lane & 7;
        const float* wp = P.W + (long long)(n0 + r0) * P.ldw + chunk * 8;
        const float* wp2 = PAIRED ? P.W2 + (long long)(n0 + r0) * P.ldw + chunk * 8 : nullptr;
        const float* xp = P.X + (long long)(t0 + r0) * P.ldx + chunk * 8;
        uint8_t* const dst = ring + r0 * 128 + ((chunk ^ (r0 & 7)) << 4);  // (rows of a thread differ by 32: the same swizzle)
        float4 v[ITEMS][2];
        auto load = [&](int i, int b) {
            const bool w = i < W_ITEMS, up = PAIRED && w && i >= W_ITEMS / 2;
            const int r = (up ? i - W_ITEMS / 2 : w ? i : i - W_ITEMS) * ROWS_PASS;
            const bool on = b < b1 && b * DS_KB + chunk * 8 < P.K && (w ? n0 + r0 + r < P.N : t0 + r0 + r < P.T);
            const float4* p = reinterpret_cast<const float4*>((up ? wp2 + r * P.ldw : w ? wp + r * P.ldw : xp + r * P.ldx) + b * DS_KB);
            v[i][0] = on ? p[0] : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][1] = on ? p[1] : make_float4(0.f, 0.f, 0.f, 0.f);
        };
#pragma unroll
        for (int i = 0; i < W_ITEMS; ++i) load(i, b0);  // the weights are constant while the stream runs
        chain_wait();
#pragma unroll
        for (int i = W_ITEMS; i < ITEMS; ++i) load(i, b0);
        uint32_t filled = 0xffffffffu;  // bit 16 stage + item: the m and l parts of this warp's rows hold (or may hold) numbers
#pragma unroll 1
        for (int b = b0; b < b1; ++b) {
            const int i0 = b - b0, s = i0 & 1;
            if (i0 >= 2 && !mbar_wait_warp(&empty_bar[s], ((i0 >> 1) - 1) & 1, &abort_flag, P.err, TC_TIMEOUT_EMPTY)) break;
            uint8_t* to = dst + s * STAGE;
            uint32_t any_m = 0, any_l = 0;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                float f[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
                load(i, b + 1);
#pragma unroll
                for (int e = 0; e < 8; e += 2) f2_unpack(f2_mul(f2_pack(f[e], f[e + 1]), f2_pack(DS_SCALE, DS_SCALE)), f[e], f[e + 1]);
                uint4* out = reinterpret_cast<uint4*>(to + (i < W_ITEMS ? i * ROWS_PASS * 128 : X_OFF + (i - W_ITEMS) * ROWS_PASS * 128));
                auto part = [&]() {
                    uint4 h;
                    h.x = ds_part(f[0], f[1]); h.y = ds_part(f[2], f[3]); h.z = ds_part(f[4], f[5]); h.w = ds_part(f[6], f[7]);
                    return h;
                };
                out[0] = part();
                if (i < W_ITEMS) {
                    // (weights that fit bf16: the parts stay as they are, zero, once they have been cleared)
                    uint32_t rest = 0;
#pragma unroll
                    for (int e = 0; e < 8; ++e) rest |= __float_as_uint(f[e]);
                    const uint32_t bit = 1u << (16 * s + i);
                    const bool some = __any_sync(0xffffffffu, (rest & 0x7fffffffu) != 0);
                    if (!some && !(filled & bit)) continue;
                    filled = some ? filled | bit : filled & ~bit;
                }
                const uint4 m = part(), l = part();
                out[PLANE / 16] = m;
                out[2 * (PLANE / 16)] = l;
                if (i < W_ITEMS) {
                    any_m |= m.x | m.y | m.z | m.w;
                    any_l |= l.x | l.y | l.z | l.w;
                }
            }
            const uint32_t parts = (__any_sync(0xffffffffu, (any_m & 0x7fff7fffu) != 0) ? 1u : 0u) | (__any_sync(0xffffffffu, (any_l & 0x7fff7fffu) != 0) ? 2u : 0u);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                w_parts[s][warp] = parts;
                mbar_arrive(&full_bar[s]);
            }
        }
    } else {
        constexpr uint32_t idesc = instr_desc_bf16(DS_ROWS, BN);
        const int quad = warp & 3, half = (warp - DS_SPLIT_WARPS) >> 2, n = b1 - b0;
        const uint32_t from = tmem + ((uint32_t)(quad * 32) << 16) + half * COLS;
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            if (warp == DS_SPLIT_WARPS) {
                const int s = i & 1;
                bool ok = mbar_wait_warp(&full_bar[s], (i >> 1) & 1, &abort_flag, P.err, TC_TIMEOUT_FULL);
                if (ok && i > 0) ok = mbar_wait_warp(&acc_empty, (i - 1) & 1, &abort_flag, P.err, TC_TIMEOUT_MISC);
                if (!ok) break;
                tc_fence_after();
                const uint32_t parts = __reduce_or_sync(0xffffffffu, lane < DS_SPLIT_WARPS ? w_parts[s][lane] : 0u);
                const uint64_t w = smem_desc_sw128(smem_u32(ring) + s * STAGE), x = smem_desc_sw128(smem_u32(ring) + s * STAGE + X_OFF);
                if (elect_one()) {
                    auto mma = [&](int to, int pw, int px, int k, uint32_t add) {
                        mma_ss(tmem + to * BUF, w + (uint64_t)(pw * (PLANE >> 4) + k * 2), x + (uint64_t)(px * (PLANE >> 4) + k * 2), idesc, add);
                    };
                    auto product = [&](int pw, int px, uint32_t add) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) mma(0, pw, px, k, k > 0 ? 1u : add);
                    };
                    // the first accumulator also takes the small products, before its large ones
                    product(0, 2, 0);
                    if (parts & 2) product(2, 0, 1);
                    if (parts & 1) product(1, 1, 1);
                    if (parts & 1) product(1, 0, 1);
                    product(0, 1, 1);
                    mma(0, 0, 0, 0, 1);
                    mma(1, 0, 0, 1, 0);
                    mma(2, 0, 0, 2, 0);
                    mma(3, 0, 0, 3, 0);
                    mma_commit(&empty_bar[s]);
                    mma_commit(&acc_full);
                }
                __syncwarp();
            }
            if (!mbar_wait_warp(&acc_full, i & 1, &abort_flag, P.err, TC_TIMEOUT_ACC)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 8) {
                uint32_t r[4][8];
#pragma unroll
                for (int q = 0; q < 4; ++q) tmem_ld8(from + q * BUF + c, r[q]);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    acc[c + j] += (__uint_as_float(r[0][j]) + __uint_as_float(r[1][j])) + (__uint_as_float(r[2][j]) + __uint_as_float(r[3][j]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty);
        }
    }
    tc_fence_before();
    __syncthreads();  // every MMA of this CTA has read its operands (the adding warps waited for the last): the ring is free
    if (warp == DS_SPLIT_WARPS) {
        tc_fence_after();
        tmem_dealloc(tmem, 4 * BUF);
    }
    if (warp >= DS_SPLIT_WARPS) {
        const int quad = warp & 3, half = (warp - DS_SPLIT_WARPS) >> 2;
        float* mine = reinterpret_cast<float*>(ring) + half * COLS * DS_ROWS + quad * 32 + lane;  // [token][feature]
#pragma unroll
        for (int j = 0; j < COLS; ++j) mine[j * DS_ROWS] = acc[j];
    }
    chain_wait();  // (C and, for results formed again, X belong to other kernels)
    if (S > 1) ds_cluster_sync();
    else __syncthreads();
    if (!abort_flag) {
        // this CTA's share of the tokens, four features per thread, the ranks' sums in order
        const int lo = BN * rank / S, hi = BN * (rank + 1) / S;
        for (int e = threadIdx.x; e < (hi - lo) * (FEATURES / 4); e += DS_THREADS) {
            const int t = lo + e / (FEATURES / 4), n = e % (FEATURES / 4) * 4;
            if (t0 + t >= P.T || n0 + n >= P.N) continue;
            // sums of four rows of the tile, formed again where they are not finite
            auto sums = [&](int row, const float* W) {
                const uint32_t at = smem_u32(ring) + (t * DS_ROWS + row) * 4;
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f), lost = v;
#pragma unroll 4
                for (int z = 0; z < S; ++z) {
                    uint32_t addr;
                    float4 q;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(at), "r"(z));
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w) : "r"(addr) : "memory");
                    ds_add(v.x, lost.x, q.x); ds_add(v.y, lost.y, q.y); ds_add(v.z, lost.z, q.z); ds_add(v.w, lost.w, q.w);
                }
                v.x += lost.x; v.y += lost.y; v.z += lost.z; v.w += lost.w;
                auto bad = [](float x) { return !(fabsf(x) < INFINITY); };
                uint32_t again = (bad(v.x) ? 1u : 0u) | (bad(v.y) ? 2u : 0u) | (bad(v.z) ? 4u : 0u) | (bad(v.w) ? 8u : 0u);
                v.x *= DS_BACK; v.y *= DS_BACK; v.z *= DS_BACK; v.w *= DS_BACK;
                if (again) v = ds_again(v, again, W + (long long)(n0 + n) * P.ldw, P.ldw, P.X + (long long)(t0 + t) * P.ldx, P.K);
                return v;
            };
            float4 v = sums(n, P.W);
            if constexpr (PAIRED) {
                const float4 u = sums(n + FEATURES, P.W2);
                auto act = [&](float g, float x) { return P.gelu ? gelu_glu_f32(g, x) : clamped_glu_f32(g, x, P.alpha, P.limit); };
                v = make_float4(act(v.x, u.x), act(v.y, u.y), act(v.z, u.z), act(v.w, u.w));
            }
            *reinterpret_cast<float4*>(P.C + (long long)(t0 + t) * P.ldc + n0 + n) = v;
        }
    }
    if (S > 1) ds_cluster_sync();  // nobody leaves while a peer reads its sums
}

// clusters of S CTAs that the chip holds at once
template <int BN, bool PAIRED>
static int ds_capacity(int S) {
    static std::mutex mu;
    static int known[64][9];  // per device
    const int guess = S == 1 ? sm_count() : sm_count() / S * 3 / 4;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return guess;
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev][S] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(S * 256);
        cfg.blockDim = dim3(DS_THREADS);
        cfg.dynamicSmemBytes = ds_smem(BN);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = S;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, dot_split_kernel<BN, PAIRED>, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = guess;
        }
        known[dev][S] = n;
    }
    return known[dev][S];
}

template <int BN, bool PAIRED>
static jsm_status ds_allow() {
    static DeviceOnce once;  // per instantiation
    JSM_CUDA_CHECK(allow_shared(once, dot_split_kernel<BN, PAIRED>, ds_smem(BN)));
    return JSM_OK;
}

// Tokens of a tile and CTAs of a cluster.  A CTA takes a bit more than a microsecond per block, most of it for the 128 rows of weights, and five to
// seven around its blocks; clusters that do not fit the chip at once wait for the first ones.  300 tokens, tokens of a tile / CTAs of a
// cluster: 1024 x 2752 96/4 24.5 us, 128/5 24.1, 64/3 26.4, 96/3 30.9, 64/4 (40 clusters, the chip holds 33) 40.7; 4096 x 512 96/1 18.6,
// 128/1 21.4, 64/1 (160 CTAs) 30.5; 33 tokens: 1024 x 1024 64/8 8.3, 96/8 8.8, 32/6 9.1, 32/8 (16 clusters, the chip holds 15) 12.8.
template <int BN, bool PAIRED>
static jsm_status ds_shape(int T, int N, int K, float* best, int* bn, int* splits) {
    constexpr float block_us = BN == 32 ? 1.04f : BN == 64 ? 1.13f : BN == 96 ? 1.2f : 1.4f, around_us = BN <= 64 ? 5.2f : BN == 96 ? 5.5f : 6.6f;
    jsm_status st = ds_allow<BN, PAIRED>();
    if (st != JSM_OK) return st;
    const int blocks = (K + DS_KB - 1) / DS_KB, tiles = ((PAIRED ? 2 : 1) * N + DS_ROWS - 1) / DS_ROWS * ((T + BN - 1) / BN);
    for (int S = 1; S <= 8 && S <= blocks; ++S) {
        const int cap = ds_capacity<BN, PAIRED>(S);
        const float cost = (float)((tiles + cap - 1) / cap) * (around_us + (S > 1 ? 0.5f : 0.0f) + (float)((blocks + S - 1) / S) * block_us);
        if (*bn == 0 || cost < *best) { *best = cost; *bn = BN; *splits = S; }
    }
    return JSM_OK;
}

template <int BN, bool PAIRED>
static jsm_status ds_launch(DotSplitParams& P, int S, cudaStream_t st) {
    P.tok_blocks = (P.T + BN - 1) / BN;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((PAIRED ? 2 : 1) * P.N + DS_ROWS - 1) / DS_ROWS * P.tok_blocks * S));
    cfg.blockDim = dim3(DS_THREADS);
    cfg.dynamicSmemBytes = ds_smem(BN);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained_launch_enabled() ? 2 : 1;
    JSM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, dot_split_kernel<BN, PAIRED>, P));
    g_launches.fetch_add(1);
    return JSM_OK;
}

// rows of 16-byte aligned fours
bool dot_split_usable(const void* X, long long ldx, const void* W, long long ldw, const void* C, long long ldc, int N, int K) {
    auto fours = [](const void* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 4 == 0; };
    return fours(X, ldx) && fours(W, ldw) && fours(C, ldc) && N % 4 == 0 && K % 8 == 0;
}

template <bool PAIRED>
static jsm_status ds_go(DotSplitParams& P, cudaStream_t st) {
    float best = 0.0f;
    int bn = 0, S = 1;
    for (auto shape : {ds_shape<128, PAIRED>, ds_shape<96, PAIRED>, ds_shape<64, PAIRED>, ds_shape<32, PAIRED>}) {
        const jsm_status s = shape(P.T, P.N, P.K, &best, &bn, &S);
        if (s != JSM_OK) return s;
    }
    return bn == 128 ? ds_launch<128, PAIRED>(P, S, st) : bn == 96 ? ds_launch<96, PAIRED>(P, S, st)
         : bn == 64 ? ds_launch<64, PAIRED>(P, S, st) : ds_launch<32, PAIRED>(P, S, st);
}
jsm_status dot_split_launch(const float* X, long long ldx, const float* W, long long ldw, float* C, long long ldc, int T, int N, int K, cudaStream_t st) {
    DotSplitParams P{X, W, nullptr, C, ldx, ldw, ldc, T, N, K, 0, tc_error_word(), 0, 0.0f, 0.0f};
    return ds_go<false>(P, st);
}
jsm_status dot_split_glu_launch(const float* X, long long ldx, const float* gate, const float* up, long long ldw, float* act, long long ldc, int T, int N, int K,
                                bool gelu, float alpha, float limit, cudaStream_t st) {
    DotSplitParams P{X, gate, up, act, ldx, ldw, ldc, T, N, K, 0, tc_error_word(), gelu ? 1 : 0, alpha, limit};
    return ds_go<true>(P, st);
}

}  // namespace jsm
