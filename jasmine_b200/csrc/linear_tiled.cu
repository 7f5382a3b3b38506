// bf16 projections of many tokens over packed weights (the layout of linear_packed.cu): Y[t, n] = sum_k X[t, k] W[n, k], the
// prompt-sized form of weight_net_t::forward (mat_net_t.hpp:38-49).
//
// What bounds it.  A prompt is tensor work: 2 T N K operations over weights that are read once.  The streaming kernel of
// linear_packed.cu takes 256 tokens per launch with the features as MMA rows, so a prompt of 2048 tokens read every matrix
// eight times, split tiles over CTAs and paid its tail (fold, transposed stores) once per 256 tokens.  Here one launch takes all
// tokens.  2048 tokens, bf16 out, 1965 MHz: 4096 x 4096 224 -> 50 us (1384 TFLOP/s), gate/up 11008 x 4096 657 -> 246 us
// (1500 TFLOP/s, 93 % of the 1619 that cuBLAS reaches at 8192^3); 512 tokens: 4096 x 4096 55 -> 19 us, 4096 x 11008 86 -> 43 us.
//
// Tile.  A pair of CTAs (cluster of two, tcgen05 cta_group::2) owns 256 tokens x BN features.  The TOKENS are the MMA rows:
// a TMEM lane is a token and a thread of the epilogue holds consecutive features of one token, so that the gate and the up
// value of a feature meet in one thread, the RMSNorm's factor is one number per thread and nothing crosses lanes.  Each CTA
// brings its 128 rows of X and half of the pair's weight rows per k-block of 64 (BN = 256: one packed tile of 128 rows each)
// with TMA; both CTAs' bytes are counted on the leader's barrier, whose thread issues the MMAs for both.
//
// Persistent: cluster c takes the tiles c, c + C, ...; the accumulator has two buffers of BN columns, so the epilogue of a tile
// overlaps the main loop of the next.  Neighbouring clusters take the token blocks of the same features: weights cross HBM once.
//
// Epilogue.  32 columns at a time go from TMEM through 4 KB of shared memory per warp (16-byte chunks, XOR swizzle: free of
// bank conflicts) and leave as whole lines: eight lanes per token.
#include "tc_utils.cuh"
#include "linear_bf16.cuh"
#include "linear_epilogue.cuh"
#include <algorithm>

namespace jsm {

using namespace tc;

constexpr int LT_BM = 256;       // tokens of a cluster's tile, 128 per CTA
constexpr int LT_EPI = 8;        // epilogue warps: two per quadrant of TMEM lanes, half of a tile's columns each
constexpr int LT_THREADS = 64 + 32 * LT_EPI;  // warp 0 TMA, warp 1 MMA, the others epilogue
constexpr int LT_KB = 2;         // k-blocks of 64 per stage: one hand-over between the threads costs about 300 cycles, more than four narrow MMAs
constexpr int LT_MAX_STAGES = 4;

struct LtParams {
    int T, N;
    int kbt;                 // k-blocks of 64
    int tok_blocks, tiles;   // tiles = tok_blocks * feature tiles of BN packed rows
    int stages;
    int epilogue, out_f32;
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

// ---- pairs of CTAs: PTX of cta_group::2 ----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void lt_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t lt_leader_addr(const void* p) {  // the same shared-memory variable in the leader CTA
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(0));
    return r;
}
// tile -> this CTA's shared memory; the bytes count on a barrier of the leader CTA
__device__ __forceinline__ void lt_load_2d(void* smem_dst, const CUtensorMap* tmap, int x, int y, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(reinterpret_cast<uint64_t>(tmap)), "r"(leader_bar), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void lt_tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void lt_tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void lt_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on `bar` of both CTAs once every MMA issued so far by this thread has completed
__device__ __forceinline__ void lt_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void lt_arrive_leader(uint32_t leader_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_bar) : "memory");
}

// TRACED: an image of its own for launches that record time stamps.
#define LT_STAMP(slot) do { if constexpr (TRACED) lin_stamp(P.trace, P.trace_ctas, slot); } while (0)
// BN: features (packed rows) per tile.  PAIRED: packed tiles of 64 gate and 64 up rows, BN / 2 outputs per token and tile.
template <int BN, bool PAIRED, bool TRACED>
__global__ void __launch_bounds__(LT_THREADS, 1)
    linear_tiled_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, LtParams P) {
    constexpr int W_ROWS = BN / 2;                 // weight rows per CTA and k-block
    constexpr uint32_t X_BYTES = 128 * 128, W_BYTES = W_ROWS * 128, STAGE = LT_KB * (X_BYTES + W_BYTES);
    constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full_bar[LT_MAX_STAGES], empty_bar[LT_MAX_STAGES];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;
    __shared__ float ssq_half[BN == 128 && !PAIRED ? 128 : 1];
    uint8_t* stage_out = tiles + P.stages * STAGE;  // 4 KB per epilogue warp

    chain_trigger();
    if (threadIdx.x == 0) LT_STAMP(0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const int stages = P.stages;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1);   // the leader's producer; the bytes of both CTAs
            mbar_init(&empty_bar[s], 1);  // the leader's MMAs, signalled in both CTAs
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * LT_EPI);  // epilogue warps of both CTAs
        }
        mbar_fence_init();
        tma_prefetch_desc(&tmap_x);
        tma_prefetch_desc(&tmap_w);
    }
    if (warp == 1) lt_tmem_alloc(&tmem_base_smem, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    lt_cluster_sync();  // both CTAs' barriers and tensor memory exist
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;

    if (warp == 0) {
        // ---- producer: the whole warp walks the stages, one elected lane issues
        auto w_row = [&](int ft) {  // first packed row of the tile that this CTA brings (of k-block 0 of its packed tile)
            if constexpr (BN == 256) return (2 * ft + (int)rank) * P.kbt * 128;
            else if constexpr (BN == 128) return ft * P.kbt * 128 + (int)rank * 64;
            else return (ft >> 1) * P.kbt * 128 + (PAIRED ? (int)rank * 64 + (ft & 1) * 32 : (ft & 1) * 64 + (int)rank * 32);
        };
        const uint32_t full_leader = lt_leader_addr(&full_bar[0]);
        struct Place { int tile, ft, tb, kb, n; };
        auto start = [&](int tile) {
            Place p;
            p.tile = tile;
            p.ft = tile / P.tok_blocks;
            p.tb = tile - p.ft * P.tok_blocks;
            p.kb = 0;
            p.n = min(LT_KB, P.kbt);
            return p;
        };
        auto next = [&](Place& p) {
            p.kb += p.n;
            if (p.kb == P.kbt) p = start(p.tile + n_clusters);
            else p.n = min(LT_KB, P.kbt - p.kb);
        };
        auto load_w = [&](int s, const Place& p) {
            if (rank == 0) mbar_expect_tx(&full_bar[s], (uint32_t)p.n * 2 * (X_BYTES + W_BYTES));
            const int row = w_row(p.ft) + p.kb * 128;
            for (int q = 0; q < p.n; ++q) lt_load_2d(tiles + s * STAGE + LT_KB * X_BYTES + q * W_BYTES, &tmap_w, 0, row + q * 128, full_leader + s * 8);
        };
        auto load_x = [&](int s, const Place& p) {
            for (int q = 0; q < p.n; ++q)
                lt_load_2d(tiles + s * STAGE + q * X_BYTES, &tmap_x, (p.kb + q) * 64, p.tb * LT_BM + (int)rank * 128, full_leader + s * 8);
        };
        // the first ring: weights before the predecessor kernel has finished, tokens once it has
        Place p = start(cluster), px = p;
        int filled = 0;
        for (; filled < stages && p.tile < P.tiles; ++filled, next(p)) {
            if (elect_one()) load_w(filled, p);
            __syncwarp();
        }
        if (lane == 0) LT_STAMP(1);
        chain_wait();
        if (lane == 0) LT_STAMP(2);
        for (int s = 0; s < filled; ++s, next(px)) {
            if (elect_one()) load_x(s, px);
            __syncwarp();
        }
        bool ok = true;
        int s = 0;
        uint32_t ph = 0;
        for (; p.tile < P.tiles; next(p)) {
            ok = mbar_wait_warp(&empty_bar[s], ph, &abort_flag, P.err, TC_TIMEOUT_EMPTY);
            if (!ok) break;
            if (elect_one()) {
                load_w(s, p);
                load_x(s, p);
            }
            __syncwarp();
            if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (!ok || abort_flag) {  // plain copies in flight land within microseconds: do not leave before them
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = instr_desc_bf16(LT_BM, BN);
            int s = 0, it = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = cluster; tile < P.tiles && ok; tile += n_clusters, ++it) {
                const int buf = it & 1;
                if (it >= 2) ok = mbar_wait_warp(&acc_empty[buf], ((it >> 1) - 1) & 1, &abort_flag, P.err, TC_TIMEOUT_MISC);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
                for (int kb = 0; kb < P.kbt; kb += LT_KB) {
                    ok = mbar_wait_warp(&full_bar[s], ph, &abort_flag, P.err, TC_TIMEOUT_FULL);
                    if (!ok) break;
                    if (it == 0 && kb == 0 && lane == 0) LT_STAMP(3);
                    tc_fence_after();
                    const uint32_t addr = smem_u32(tiles + s * STAGE);
                    const uint64_t a_desc = smem_desc_sw128(addr), b_desc = smem_desc_sw128(addr + LT_KB * X_BYTES);
                    const bool both = kb + 1 < P.kbt;
                    if (elect_one()) {
#pragma unroll
                        for (int q = 0; q < LT_KB; ++q)
                            if (q == 0 || both)
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    lt_mma(d_tmem, a_desc + (uint64_t)(q * (X_BYTES >> 4) + k * 2), b_desc + (uint64_t)(q * (W_BYTES >> 4) + k * 2), idesc,
                                           (kb > 0 || q > 0 || k > 0) ? 1u : 0u);
                        lt_commit(&empty_bar[s]);
                    }
                    __syncwarp();
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
                if (ok && elect_one()) lt_commit(&acc_full[buf]);
                __syncwarp();
            }
            if (lane == 0) LT_STAMP(4);
        }
    } else {
        const int quad = warp & 3;  // TMEM lanes this warp reads
        const int half = (warp - 2) >> 2;  // which half of the columns
        uint8_t* out_smem = stage_out + (warp - 2) * 4096;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t empty_leader[2] = {lt_leader_addr(&acc_empty[0]), lt_leader_addr(&acc_empty[1])};
        const int c4 = (lane & 7) * 4, r4 = lane >> 3;  // the place a lane reads back: 4 columns of every fourth row
        chain_wait();
        int it = 0;
        bool ok = true;  // a warp that gave up a wait walks on without work: it still meets the others at the barriers of the row statistics
        for (int tile = cluster; tile < P.tiles; tile += n_clusters, ++it) {
            const int ft = tile / P.tok_blocks, tb = tile - ft * P.tok_blocks;
            const int t0 = tb * LT_BM + (int)rank * 128 + quad * 32;  // first token of this warp
            const int buf = it & 1;
            float scale = 1.0f;
            if (P.ssq_in) {  // fused RMSNorm: the per-tile sums of squares of the token's row, added in tile order
                float q = 0.0f;
                if (t0 + lane < P.T)
                    for (int j = 0; j < P.ssq_in_tiles; ++j) q += __ldcg(P.ssq_in + (size_t)j * P.ssq_stride + t0 + lane);
                scale = rsqrtf(q * P.inv_d + P.eps);
            }
            ok = ok && mbar_wait(&acc_full[buf], (it >> 1) & 1, &abort_flag, P.err, TC_TIMEOUT_ACC);
            tc_fence_after();
            const uint32_t acc = lane_addr + (uint32_t)(buf * BN);
            constexpr int CHUNKS = PAIRED ? BN / 64 : BN / 32, MINE = CHUNKS > 1 ? CHUNKS / 2 : 1;
            const int c_end = ok && (CHUNKS > 1 || half == 0) ? (half + 1) * MINE : 0;
            float ssq[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) ssq[k] = 0.0f;
#pragma unroll 1
            for (int c = half * MINE; c < c_end; ++c) {
                // outputs n0 .. n0 + 31 of the tokens t0 .. t0 + 31
                const int n0 = ft * (PAIRED ? BN / 2 : BN) + c * 32, n = n0 + c4;
                const bool n_ok = n < P.N;
                uint2 rr[8];
                if (!PAIRED && P.epilogue == LIN_RESIDUAL)
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int t = t0 + 4 * k + r4;
                        rr[k] = n_ok && t < P.T ? *reinterpret_cast<const uint2*>(P.R + (size_t)t * P.N + n) : make_uint2(0u, 0u);
                    }
                uint32_t r[32];
                if constexpr (PAIRED) {
                    uint32_t up[32];
                    // tiles of 128 packed rows: 64 gate columns, then their 64 up columns (BN = 64: 32 and 32)
                    const int g = BN == 64 ? 0 : (c >> 1) * 128 + (c & 1) * 32;
                    tmem_ld32(acc + g, r);
                    tmem_ld32(acc + g + (BN == 64 ? 32 : 64), up);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float gv = __uint_as_float(r[j]) * scale, uv = __uint_as_float(up[j]) * scale;
                        const float v = P.epilogue == LIN_CLAMPED_GLU ? pk_clamped_glu(gv, uv, P.glu_alpha, P.glu_limit)
                                        : P.epilogue == LIN_GELU_GLU  ? pk_gelu_glu(gv, uv)
                                                                      : pk_silu(gv) * uv;
                        r[j] = __float_as_uint(v);
                    }
                } else {
                    tmem_ld32(acc + c * 32, r);
                    tmem_ld_wait();
                    if (P.ssq_in)
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * scale);
                }
                if (c == c_end - 1) {  // the accumulator is read: the MMAs of the tile after the next may have it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) lt_arrive_leader(empty_leader[buf]);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<uint4*>(out_smem + lane * 128 + ((j ^ (lane & 7)) * 16)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                __syncwarp();
                const float4 bias = !PAIRED && P.bias && n_ok ? *reinterpret_cast<const float4*>(P.bias + n) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int row = 4 * k + r4, t = t0 + row;
                    float4 v = *reinterpret_cast<const float4*>(out_smem + row * 128 + (((lane & 7) ^ (row & 7)) * 16));
                    if constexpr (!PAIRED) {
                        v.x += bias.x; v.y += bias.y; v.z += bias.z; v.w += bias.w;
                        if (P.epilogue == LIN_RELU) {
                            v.x = fmaxf(v.x, 0.0f); v.y = fmaxf(v.y, 0.0f); v.z = fmaxf(v.z, 0.0f); v.w = fmaxf(v.w, 0.0f);
                        } else if (P.epilogue == LIN_GELU) {
                            v.x = pk_gelu(v.x); v.y = pk_gelu(v.y); v.z = pk_gelu(v.z); v.w = pk_gelu(v.w);
                        } else if (P.epilogue == LIN_RESIDUAL) {
                            v.x += bf16lo(rr[k].x); v.y += bf16hi(rr[k].x); v.z += bf16lo(rr[k].y); v.w += bf16hi(rr[k].y);
                        }
                    }
                    if (n_ok && t < P.T) {
                        if (P.out_f32) {
                            *reinterpret_cast<float4*>(static_cast<float*>(P.Y) + (size_t)t * P.N + n) = v;
                        } else {
                            const uint2 o = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
                            *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(P.Y) + (size_t)t * P.N + n) = o;
                            if (!PAIRED && P.ssq_out) {
                                const float a = bf16lo(o.x), b = bf16hi(o.x), d = bf16lo(o.y), e = bf16hi(o.y);
                                ssq[k] += (a * a + b * b) + (d * d + e * e);
                            }
                        }
                    }
                }
                __syncwarp();  // the staging tile is free again
            }
            if (ok && CHUNKS == 1 && half == 1) {  // (nothing of this tile to read)
                __syncwarp();
                if (lane == 0) lt_arrive_leader(empty_leader[buf]);
            }
            if (!PAIRED && BN >= 128 && P.ssq_out) {  // one number per token and 128 features
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) ssq[k] += __shfl_xor_sync(0xffffffffu, ssq[k], o);
                if (BN == 128) {  // two warps share the 128 features
                    if (half == 1 && (lane & 7) == 0)
#pragma unroll
                        for (int k = 0; k < 8; ++k) ssq_half[quad * 32 + 4 * k + r4] = ssq[k];
                    asm volatile("bar.sync 1, %0;" ::"n"(32 * LT_EPI) : "memory");
                    if (half == 0 && (lane & 7) == 0)
#pragma unroll
                        for (int k = 0; k < 8; ++k) ssq[k] += ssq_half[quad * 32 + 4 * k + r4];
                    asm volatile("bar.sync 1, %0;" ::"n"(32 * LT_EPI) : "memory");  // (the next tile writes it again)
                }
                const int tile128 = BN == 256 ? 2 * ft + half : ft;
                if (ok && (BN == 256 || half == 0) && (lane & 7) == 0 && tile128 * 128 < P.N)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (t0 + 4 * k + r4 < P.T) P.ssq_out[(size_t)tile128 * P.ssq_stride + t0 + 4 * k + r4] = ssq[k];
            }
            if (warp == 2 && lane == 0) LT_STAMP(it == 0 ? 5 : 6);
        }
    }
    tc_fence_before();
    __syncwarp();
    __syncthreads();
    lt_cluster_sync();  // nobody leaves while the pair's MMAs, copies or arrivals may still reach its shared memory
    if (warp == 1) {
        tc_fence_after();
        lt_tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0) LT_STAMP(7);
}

template <int BN, bool PAIRED, bool TRACED = false>
static jsm_status launch_tiled(const PackedArgs& a, LtParams& P, int n_tiles, cudaStream_t st) {
    if (!TRACED && (P.trace = linear_trace_next(&P.trace_ctas))) return launch_tiled<BN, PAIRED, true>(a, P, n_tiles, st);
    constexpr int STAGE = LT_KB * (128 * 128 + BN / 2 * 128);
    P.stages = std::min(LT_MAX_STAGES, 192 * 1024 / STAGE);
    const size_t smem = (size_t)P.stages * STAGE + LT_EPI * 4096 + 1024;
    const int f_tiles = BN == 256 ? (n_tiles + 1) / 2 : BN == 128 ? n_tiles : 2 * n_tiles;
    P.tiles = P.tok_blocks * f_tiles;
    CUtensorMap mx, mw;
    jsm_status s = make_tmap_bf16_2d(&mx, a.X, (uint64_t)a.T, (uint64_t)a.K, (uint64_t)(a.x_row_stride > 0 ? a.x_row_stride : a.K), 128, 64);
    if (s != JSM_OK) return s;
    // the packed image as rows of 64 elements; it already has the shared-memory order
    s = make_tmap_bf16_2d(&mw, a.Wp, (uint64_t)n_tiles * P.kbt * 128, 64, 64, BN / 2, 64, false);
    if (s != JSM_OK) return s;
    static DeviceOnce once;  // per instantiation
    JSM_CUDA_CHECK(allow_shared(once, linear_tiled_kernel<BN, PAIRED, TRACED>, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * std::min(P.tiles, sm_count() / 2));
    cfg.blockDim = dim3(LT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.chained && chained_launch_enabled() ? 2 : 1;
    JSM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, linear_tiled_kernel<BN, PAIRED, TRACED>, mx, mw, P));
    g_launches.fetch_add(1);
    return JSM_OK;
}

// Arguments checked by linear_packed_tokens.
jsm_status linear_tiled_launch(const PackedArgs& a, cudaStream_t st) {
    const int paired = a.epilogue == LIN_SILU_MUL || a.epilogue == LIN_CLAMPED_GLU || a.epilogue == LIN_GELU_GLU;
    LtParams P;
    int n_tiles;
    pk_dims(a.N, a.K, paired, &n_tiles, &P.kbt);
    P.T = a.T; P.N = a.N;
    P.tok_blocks = (a.T + LT_BM - 1) / LT_BM;
    P.epilogue = a.epilogue; P.out_f32 = a.out_f32 ? 1 : 0;
    P.bias = a.bias; P.R = static_cast<const __nv_bfloat16*>(a.R); P.Y = a.Y;
    P.ssq_in = a.ssq_in; P.ssq_in_tiles = a.ssq_in_tiles; P.ssq_stride = a.ssq_stride > 0 ? a.ssq_stride : a.T;
    P.inv_d = 1.0f / (float)a.K; P.eps = a.eps; P.ssq_out = a.ssq_out;
    P.glu_alpha = a.glu_alpha; P.glu_limit = a.glu_limit;
    P.err = tc_error_word();
    // The widest tile moves the fewest bytes per operation, a narrower one fills the last wave of clusters better.  Time of a wave
    // relative to BN = 256, measured over 64 k-blocks: 22.5, 12.6 and 11.5 us (narrow tiles: bound by the hand-over of the stages).
    const int clusters = sm_count() / 2;
    auto waves = [&](int f_tiles) { return (P.tok_blocks * f_tiles + clusters - 1) / clusters; };
    const float c256 = 1.0f * waves((n_tiles + 1) / 2), c128 = 0.56f * waves(n_tiles);
    const float c64 = a.ssq_out ? 1e9f : 0.51f * waves(2 * n_tiles);  // (statistics come per 128 features)
    const int bn = c64 < c128 && c64 < c256 ? 64 : c128 < c256 ? 128 : 256;
    if (paired)
        return bn == 256 ? launch_tiled<256, true>(a, P, n_tiles, st) : bn == 128 ? launch_tiled<128, true>(a, P, n_tiles, st) : launch_tiled<64, true>(a, P, n_tiles, st);
    return bn == 256 ? launch_tiled<256, false>(a, P, n_tiles, st) : bn == 128 ? launch_tiled<128, false>(a, P, n_tiles, st) : launch_tiled<64, false>(a, P, n_tiles, st);
}

}  // namespace jsm
