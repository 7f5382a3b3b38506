// fp32 contraction with the summation order of the reference's mat_dot_t
// (mat_express_t.hpp:730-736): each output element is s = 0; s += a(i,k) * b(k,j)
// for k ascending, multiply and add rounded separately.  Used for the
// reference-exact fp32 paths (small models, parity tests) and, in another order, for few
// tokens of f32 models; their other products run on the tensor cores (dot_split.cu).
#include "common.cuh"
#include "mma_utils.cuh"
#include "tc_utils.cuh"

namespace jsm {

using tc::smem_u32;

struct MatD {
    const float* p;
    int rows, cols;
    long long rs, cs;
};

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752440f)); }

// Tile.  128 threads own TMM * 8 rows x TNN * 16 columns, TMM x TNN outputs each (rows ty + 8 i, columns tx + 16 j).  Blocks of
// 32 products are staged [row or column][k] by asynchronous copies, so that a thread reads four of them with one load and the
// four rows or eight columns of a quarter warp lie in different banks (pitch 36).
constexpr int DOT_THREADS = 128, DOT_KB = 32, DOT_PITCH = DOT_KB + 4;
constexpr int dot_stages(int tnn) { return tnn == 1 ? 8 : 4; }
constexpr int dot_smem(int tmm, int tnn) { return dot_stages(tnn) * (8 * tmm + 16 * tnn) * DOT_PITCH * 4; }

// One thread's part in staging 32 products' worth of ROWS rows of an operand (row stride rs, stride ks along the products), zeros where
// there is nothing.  Its first address and its bounds are worked out once; a warp walks
//   VEC  contiguous products in 16-byte aligned rows: four products of every 16th row per thread
//   ROW  contiguous rows (a transposed operand): eight rows by four products at a time, whole sectors of memory and all banks
//   ANY  other strides, or contiguous products off alignment: 32 products of every fourth row
// (With addresses worked out per element of four bytes a transposed operand cost as many instructions as a sixth of the products.  In the
// reference's order, us, both operands transposed / the second / none: 1024 x 4096 x 128 87 / 83 / 73, here 79 / 75 / 73; 512 x 512 x 512
// 46 / 35 / 26, here 33 / 30 / 26.)
enum DotWalk { DOT_VEC, DOT_ROW, DOT_ANY };
template <int ROWS>
struct DotLoader {
    static constexpr int WARPS = DOT_THREADS / 32, STEP = DOT_THREADS / (DOT_KB / 4), OCTETS = ROWS / 8;
    static_assert(ROWS % STEP == 0 && (OCTETS == 2 || OCTETS == 2 * WARPS), "whole passes");
    const float *base, *p;  // the operand; first element of the thread
    long long rs, ks;
    int rows, left, walk;   // rows from the thread's first on, products of the operand from its first on
    uint32_t dst;           // offset of the thread's first element in a stage
    __device__ __forceinline__ DotLoader(const float* base, int row0, int rows, long long rs, long long ks, int K, int walk)
        : base(base), rs(rs), ks(ks), walk(walk) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        int r, x;
        if (walk == DOT_VEC) { r = threadIdx.x / (DOT_KB / 4); x = threadIdx.x % (DOT_KB / 4) * 4; }
        else if (walk == DOT_ROW) { r = warp % OCTETS * 8 + lane % 8; x = warp / OCTETS * 4 + lane / 8; }
        else { r = warp; x = lane; }
        p = base + (row0 + r) * rs + x * ks;
        this->rows = rows - row0 - r;
        left = K - x;
        dst = (r * DOT_PITCH + x) * 4;
    }
    __device__ __forceinline__ void operator()(uint32_t stage, int k0) const {
        const int n = left - k0;  // products left
        const uint32_t to = stage + dst;
        if (walk == DOT_VEC) {
            const int bytes_row = min(max(n, 0), 4) * 4;
            const float* src = p + k0;
#pragma unroll
            for (int i = 0; i < ROWS / STEP; ++i) {
                const int bytes = i * STEP < rows ? bytes_row : 0;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + i * STEP * DOT_PITCH * 4),
                             "l"(reinterpret_cast<uint64_t>(bytes ? src : base)), "r"(bytes)
                             : "memory");
                src += STEP * rs;
            }
        } else if (walk == DOT_ROW) {
            const float* src = p + k0 * ks;
            constexpr int RUN = OCTETS > WARPS ? OCTETS / WARPS : 1, KSTEP = OCTETS > WARPS ? 4 : WARPS / OCTETS * 4;  // octets of rows per step of KSTEP products
#pragma unroll
            for (int x = 0; x < DOT_KB; x += KSTEP) {
#pragma unroll
                for (int i = 0; i < RUN; ++i) {
                    const bool on = x < n && i * WARPS * 8 < rows;
                    cp_async4(to + (i * WARPS * 8 * DOT_PITCH + x) * 4, on ? src + i * WARPS * 8 : base, on);
                }
                src += KSTEP * ks;
            }
        } else {
            const float* src = p + k0 * ks;
#pragma unroll 4
            for (int i = 0; i < ROWS / WARPS; ++i) {
                const bool on = n > 0 && i * WARPS < rows;
                cp_async4(to + i * WARPS * DOT_PITCH * 4, on ? src : base, on);
                src += WARPS * rs;
            }
        }
    }
};

// Before, one 64 x 64 tile per CTA staged element by element: 64 x 128 x 128 took 27 us, 300 x 1024 x 2752 (f32 model) 182 us.
// What bounds it: with few outputs the chain of K dependent additions and the launch, with many the fp32 pipe (two instructions
// per product in the reference's order, one per two products otherwise).
// ORDERED: the reference's summation order (see above).  The zeros behind the last product change nothing: a sum that starts
// at +0 never becomes -0.
// Otherwise: even and odd products of a block of 32 form two chains of fused multiply-adds (packed pairs), which join the total
// once per block; a cluster of CTAs shares the products of a tile (whole blocks each) and adds its totals in rank order.
template <bool ORDERED, int TMM, int TNN>
__global__ void __launch_bounds__(DOT_THREADS, TMM == 8 ? 3 : 4) dot_f32_kernel(MatD A, MatD B, MatD bias, int has_bias, int epilogue, MatD R,
                                                              float* Cp, long long crs, long long ccs, int M, int N, int K, int walk_a, int walk_b) {
    constexpr int BM = 8 * TMM, BN = 16 * TNN, STAGES = dot_stages(TNN), STAGE = (BM + BN) * DOT_PITCH;
    static_assert(STAGES * STAGE >= BM * BN, "the totals of a tile are exchanged through the ring");
    extern __shared__ __align__(16) float dot_ring[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int splits = ORDERED ? 1 : gridDim.z, rank = ORDERED ? 0 : blockIdx.z;
    const int blocks = (K + DOT_KB - 1) / DOT_KB, b0 = (int)((long long)blocks * rank / splits), mine = (int)((long long)blocks * (rank + 1) / splits) - b0;
    const uint32_t ring = smem_u32(dot_ring);
    const DotLoader<BM> load_a(A.p, m0, M, A.rs, A.cs, K, walk_a);
    const DotLoader<BN> load_b(B.p, n0, N, B.cs, B.rs, K, walk_b);
    auto stage_a = [&](int i) { load_a(ring + (i % STAGES) * STAGE * 4, (b0 + i) * DOT_KB); };
    auto stage_b = [&](int i) { load_b(ring + ((i % STAGES) * STAGE + BM * DOT_PITCH) * 4, (b0 + i) * DOT_KB); };
    if (!ORDERED) chain_trigger();
#pragma unroll 1
    for (int i = 0; i < STAGES - 1; ++i) {
        if (i < mine) {
            stage_a(i);
            stage_b(i);
        }
        cp_async_commit();
    }
    float acc[TMM][TNN];
#pragma unroll
    for (int i = 0; i < TMM; ++i)
#pragma unroll
        for (int j = 0; j < TNN; ++j) acc[i][j] = 0.0f;
#pragma unroll 1
    for (int b = 0; b < mine; ++b) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();  // block b is here, and everybody is done with block b - 1, whose place is filled again
        if (b + STAGES - 1 < mine) {
            stage_a(b + STAGES - 1);
            stage_b(b + STAGES - 1);
        }
        cp_async_commit();
        const float *as = dot_ring + (b % STAGES) * STAGE + ty * DOT_PITCH, *bs = dot_ring + (b % STAGES) * STAGE + (BM + tx) * DOT_PITCH;
        if constexpr (ORDERED) {
#pragma unroll 2
            for (int k = 0; k < DOT_KB; k += 4) {
                float4 x[TMM], y[TNN];
#pragma unroll
                for (int i = 0; i < TMM; ++i) x[i] = *reinterpret_cast<const float4*>(as + i * 8 * DOT_PITCH + k);
#pragma unroll
                for (int j = 0; j < TNN; ++j) y[j] = *reinterpret_cast<const float4*>(bs + j * 16 * DOT_PITCH + k);
#pragma unroll
                for (int i = 0; i < TMM; ++i)
#pragma unroll
                    for (int j = 0; j < TNN; ++j) {
                        float s = acc[i][j];
                        s = __fadd_rn(s, __fmul_rn(x[i].x, y[j].x));
                        s = __fadd_rn(s, __fmul_rn(x[i].y, y[j].y));
                        s = __fadd_rn(s, __fmul_rn(x[i].z, y[j].z));
                        acc[i][j] = __fadd_rn(s, __fmul_rn(x[i].w, y[j].w));
                    }
            }
        } else {
            uint64_t part[TMM][TNN];  // (a product's operands are a pass over all outputs apart: no instruction waits for the one before it)
#pragma unroll
            for (int k = 0; k < DOT_KB; k += 4) {
                ulonglong2 x[TMM], y[TNN];
#pragma unroll
                for (int i = 0; i < TMM; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(as + i * 8 * DOT_PITCH + k);
#pragma unroll
                for (int j = 0; j < TNN; ++j) y[j] = *reinterpret_cast<const ulonglong2*>(bs + j * 16 * DOT_PITCH + k);
#pragma unroll
                for (int i = 0; i < TMM; ++i)
#pragma unroll
                    for (int j = 0; j < TNN; ++j) part[i][j] = k == 0 ? f2_mul(x[i].x, y[j].x) : f2_fma(x[i].x, y[j].x, part[i][j]);
#pragma unroll
                for (int i = 0; i < TMM; ++i)
#pragma unroll
                    for (int j = 0; j < TNN; ++j) part[i][j] = f2_fma(x[i].y, y[j].y, part[i][j]);
            }
#pragma unroll
            for (int i = 0; i < TMM; ++i)
#pragma unroll
                for (int j = 0; j < TNN; ++j) {
                    float even, odd;
                    f2_unpack(part[i][j], even, odd);
                    acc[i][j] += even + odd;
                }
        }
    }
    if constexpr (ORDERED) {
#pragma unroll
        for (int i = 0; i < TMM; ++i)
#pragma unroll
            for (int j = 0; j < TNN; ++j) {
                const int m = m0 + ty + 8 * i, n = n0 + tx + 16 * j;
                if (m < M && n < N) {
                    float v = acc[i][j];
                    if (has_bias) v = __fadd_rn(v, bias.p[(m < bias.rows ? m : m % bias.rows) * bias.rs + (n < bias.cols ? n : n % bias.cols) * bias.cs]);
                    if (epilogue == 1) v = v > 0.0f ? v : 0.0f * v;
                    else if (epilogue == 2) v = gelu_f(v);
                    else if (epilogue == 3) v = __fadd_rn(v, R.p[(m < R.rows ? m : m % R.rows) * R.rs + (n < R.cols ? n : n % R.cols) * R.cs]);
                    Cp[m * crs + n * ccs] = v;
                }
            }
    } else {
        cp_async_wait<0>();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TMM; ++i)
#pragma unroll
            for (int j = 0; j < TNN; ++j) dot_ring[(ty + 8 * i) * BN + tx + 16 * j] = acc[i][j];
        if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        else __syncthreads();
        // this CTA's share of the rows (8 TMM >= splits, both powers of two)
        const int rows = BM / splits;
        for (int e = threadIdx.x; e < rows * BN; e += DOT_THREADS) {
            const int r = rank * rows + e / BN, c = e % BN;
            float v = 0.0f;
            if (splits == 1) v = dot_ring[r * BN + c];
            else
                for (int s = 0; s < splits; ++s) {
                    uint32_t addr;
                    float t;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(ring + (r * BN + c) * 4), "r"(s));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t) : "r"(addr) : "memory");
                    v += t;
                }
            if (m0 + r < M && n0 + c < N) Cp[(m0 + r) * crs + (n0 + c) * ccs] = v;
        }
        if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

static MatD to_d(const jsm_mat& m) {
    MatD d;
    d.p = reinterpret_cast<const float*>(m.data);
    d.rows = m.rows; d.cols = m.cols; d.rs = m.row_stride; d.cs = m.col_stride;
    return d;
}

static int dot_walk(const float* p, long long rs, long long ks) {
    return ks == 1 && rs % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0 ? DOT_VEC : rs == 1 ? DOT_ROW : DOT_ANY;
}

template <bool ORDERED, int TMM, int TNN>
static jsm_status dot_launch(const MatD& A, const MatD& B, const MatD* bias, int epilogue, const MatD* R, float* C, long long crs, long long ccs, int splits,
                             cudaStream_t st) {
    constexpr int smem = dot_smem(TMM, TNN);
    static DeviceOnce once;  // per instantiation
    JSM_CUDA_CHECK(allow_shared(once, dot_f32_kernel<ORDERED, TMM, TNN>, smem));
    const MatD none{nullptr, 1, 1, 0, 0};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((B.cols + 16 * TNN - 1) / (16 * TNN), (A.rows + 8 * TMM - 1) / (8 * TMM), splits);
    cfg.blockDim = dim3(DOT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];  // (plain stream order: see launch_spread)
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = splits;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    JSM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, dot_f32_kernel<ORDERED, TMM, TNN>, A, B, bias ? *bias : none, bias ? 1 : 0, epilogue, R ? *R : none, C, crs, ccs, A.rows,
                                      B.cols, A.cols, dot_walk(A.p, A.rs, A.cs), dot_walk(B.p, B.cs, B.rs)));
    g_launches.fetch_add(1);
    return JSM_OK;
}

bool dot_split_usable(const void* X, long long ldx, const void* W, long long ldw, const void* C, long long ldc, int N, int K);
jsm_status dot_split_launch(const float* X, long long ldx, const float* W, long long ldw, float* C, long long ldc, int T, int N, int K, cudaStream_t st);

// whether the tensor cores take X . W^T (below): rows of aligned fours
bool dot_f32_splits(const void* X, long long ldx, const void* W, long long ldw, const void* C, long long ldc, int T, int N, int K) {
    return (T > 32 || (long long)N * K >= 1 << 20) && dot_split_usable(X, ldx, W, ldw, C, ldc, N, K);
}

// C = A . B in fp32 without the reference's order (operands as in jsm_dot_f32, checked by the caller).  Rows of aligned fours go to the tensor cores
// (dot_split.cu) from 33 rows of A on, and below that from a million weights on.  The line lies between what a launch takes by itself and what it takes
// in a chain, where its start lies behind its predecessor (us, here / there; by itself, then back to back: 8 rows, 512 x 512 5.0 / 7.5, 6.2 / 5.4; 1024 x
// 1024 7.4 / 8.5, 8.2 / 7.2; 4096 x 512 9.3 / 8.5, 10.3 / 7.7; 2752 x 1024 13.9 / 9.8, 15.5 / 9.4; 32 rows, 512 x 512 5.8 / 7.7, 6.2 / 5.8; 1024 x 1024
// 8.8 / 8.9, 10.3 / 7.7; 2752 x 1024 21.6 / 10.4, 22.6 / 9.8; weights of 24 bits).  33 rows, in the 64 x 64 tiles that this kernel had for them, back to
// back: 64 x 64 7.7 / 4.1, 512 x 512 6.5 / 5.9.
// The others take 16 x 64 tiles, whose products are shared by as many CTAs as even out the multiprocessors' loads: rounds of
// CTAs times blocks of products each, and about four blocks' time for a CTA's start and end.
jsm_status dot_f32_launch(const jsm_mat& A, const jsm_mat& B, const jsm_mat& Cm, cudaStream_t st) {
    float* C = reinterpret_cast<float*>(Cm.data);
    if (A.col_stride == 1 && B.row_stride == 1 && Cm.col_stride == 1 &&
        dot_f32_splits(A.data, A.row_stride, B.data, B.col_stride, C, Cm.row_stride, A.rows, B.cols, A.cols))
        return dot_split_launch(static_cast<const float*>(A.data), A.row_stride, static_cast<const float*>(B.data), B.col_stride, C, Cm.row_stride, A.rows,
                                B.cols, A.cols, st);
    const int tiles = (B.cols + 63) / 64 * ((A.rows + 15) / 16), blocks = (A.cols + DOT_KB - 1) / DOT_KB;
    int splits = 1;
    long long best = -1;
    for (int s = 1; s <= 8 && s <= blocks; s *= 2) {
        const long long cost = (long long)((tiles * s + sm_count() - 1) / sm_count()) * ((blocks + s - 1) / s + 4);
        if (best < 0 || cost < best) { best = cost; splits = s; }
    }
    return dot_launch<false, 2, 4>(to_d(A), to_d(B), nullptr, 0, nullptr, C, Cm.row_stride, Cm.col_stride, splits, st);
}

// whether the spans of memory of two matrices meet
static bool dot_overlap(const jsm_mat& a, const jsm_mat& b) {
    auto span = [](const jsm_mat& m, uintptr_t& lo, uintptr_t& hi) {
        const long long r = (m.rows - 1) * (long long)m.row_stride * 4, c = (m.cols - 1) * (long long)m.col_stride * 4;
        lo = reinterpret_cast<uintptr_t>(m.data) + (r < 0 ? r : 0) + (c < 0 ? c : 0);
        hi = reinterpret_cast<uintptr_t>(m.data) + (r > 0 ? r : 0) + (c > 0 ? c : 0) + 4;
    };
    uintptr_t a0, a1, b0, b1;
    span(a, a0, a1);
    span(b, b0, b1);
    return a0 < b1 && b0 < a1;
}

}  // namespace jsm

using namespace jsm;

extern "C" jsm_status jsm_dot_f32(jsm_mat A, jsm_mat B, const jsm_mat* bias, int epilogue, const jsm_mat* R, jsm_mat Cm,
                                  void* stream) {
    if (A.cols != B.rows)
        JSM_FAIL(JSM_INVALID_ARG, "mat_dot_t: inner dimensions do not match for dot product (%d x %d . %d x %d)", A.rows,
                 A.cols, B.rows, B.cols);
    if (A.dtype != JSM_F32 || B.dtype != JSM_F32 || Cm.dtype != JSM_F32) JSM_FAIL(JSM_UNSUPPORTED, "jsm_dot_f32: f32 only");
    if (Cm.rows != A.rows || Cm.cols != B.cols)
        JSM_FAIL(JSM_SHAPE, "jsm_dot_f32: output is %d x %d, product is %d x %d", Cm.rows, Cm.cols, A.rows, B.cols);
    if (epilogue < 0 || epilogue > 3 || (epilogue == 3 && !R)) JSM_FAIL(JSM_INVALID_ARG, "jsm_dot_f32: epilogue %d", epilogue);
    if (A.rows == 0 || B.cols == 0) return JSM_OK;
    if (!A.data || !B.data || !Cm.data) JSM_FAIL(JSM_INVALID_ARG, "jsm_dot_f32: null operand");
    if ((bias && (bias->dtype != JSM_F32 || !bias->data || bias->rows <= 0 || bias->cols <= 0)) ||
        (R && (R->dtype != JSM_F32 || !R->data || R->rows <= 0 || R->cols <= 0)))
        JSM_FAIL(JSM_INVALID_ARG, "jsm_dot_f32: bad bias / residual operand");
    MatD bd, rd;
    if (bias) bd = to_d(*bias);
    if (R) rd = to_d(*R);
    const MatD *pb = bias ? &bd : nullptr, *pr = R ? &rd : nullptr;
    float* C = reinterpret_cast<float*>(Cm.data);
    // 64 x 64 tiles once they occupy half of the multiprocessors, 16 x 16 tiles (one output pair per thread) below.  A product of one 64 x 64
    // tile may lie in an operand's memory (x <- x W): its one CTA has read everything before it writes, several would not.
    const long long tiles = (long long)((Cm.cols + 63) / 64) * ((Cm.rows + 63) / 64);
    if (tiles * 2 > sm_count() || (tiles == 1 && (dot_overlap(Cm, A) || dot_overlap(Cm, B))))
        return dot_launch<true, 8, 4>(to_d(A), to_d(B), pb, epilogue, pr, C, Cm.row_stride, Cm.col_stride, 1, as_stream(stream));
    return dot_launch<true, 2, 1>(to_d(A), to_d(B), pb, epilogue, pr, C, Cm.row_stride, Cm.col_stride, 1, as_stream(stream));
}
