// out[M,N] (=|+=) a[M,K] . w[N,K]^T (+ bias): the plain matrix product.
//
// Float32 multiply-adds only, a fixed summation order over k for every output element (it depends on the sizes, never on
// the values), any sizes, any mix of float32 / bfloat16 operands.  It is the whole float32 path's product and the
// comparison for the tensor-core kernels, in the way the reference keeps portable kernels beside its vector ones
// (src/kern_generic.c:84-91 beside src/kern_avx2.c:79-95; call shape src/model.c:419-425).
//
// Two kernels.  Up to ROWS_MAX rows (single tokens) the product only streams the weights: a warp takes ROWS_N weight rows
// at a time, sixteen bytes a lane, and the sum over the lanes comes last.  More rows are bound by the float32 units:
// tiles of registers over double-buffered shared memory, the next piece of k on its way from global memory while one
// is multiplied, two neighbouring features an instruction (fma.rn.f32x2: each half rounds as an fma of its own, and the
// units stay fed while other instructions issue).  Where the tiles are fewer than the SMs the inner dimension is cut
// among the CTAs of a cluster, and each of them sums a share of the tile's rows over the cluster's shared memories, in the
// order of the slices: no workspace, no second pass over memory.
// Measured (B200, float32; one 64 x 64 tile of 16 k for every size before): see the rule in hfb_linear_plain.
#include "common.cuh"

static thread_local cudaError_t g_launch_err = cudaSuccess;      // what the last launch of this thread returned

namespace hfb {

// ---- many rows: tiles of BM x BN, TM x TN a thread -------------------------------------------------------------------
constexpr int TK = 16;               // of k a stage
constexpr int MAX_SPLITS = 8;        // CTAs of a cluster

__device__ __forceinline__ unsigned long long pack2(float x, float y)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long &acc, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Four consecutive values of a row from k on, zeros from K on.  VEC: K is a multiple of 4 and the rows are aligned to four values.
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T *row, int k, int K, bool live)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!live) return v;
    if (VEC) {
        if (k < K) {
            if constexpr (sizeof(T) == 4) {
                v = *(const float4 *)(row + k);
            } else {
                const uint2 u = *(const uint2 *)(row + k);
                const float2 lo = __bfloat1622float2(*(const __nv_bfloat162 *)&u.x), hi = __bfloat1622float2(*(const __nv_bfloat162 *)&u.y);
                v = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
    } else {
        if (k < K) v.x = to_f32(row[k]);
        if (k + 1 < K) v.y = to_f32(row[k + 1]);
        if (k + 2 < K) v.z = to_f32(row[k + 2]);
        if (k + 3 < K) v.w = to_f32(row[k + 3]);
    }
    return v;
}

template <int BM, int BN> constexpr int tile_floats()
{
    const int stages = 2 * TK * (BM + 4 + BN + 4), sums = BM * BN;
    return stages > sums ? stages : sums;
}

template <typename TA, typename TW, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), BM == 128 ? 2 : 1)
linear_tile_kernel(const TA *__restrict__ a, const TW *__restrict__ w, const void *bias, int bias_dt, void *out, int out_dt,
                   int accumulate, int M, int N, int K, int tiles_m, int k_slice)
{
    constexpr int THREADS = (BM / TM) * (BN / TN), TX = BN / TN;
    // pieces of four values a thread fetches (of a tile of few rows only the first threads have one)
    constexpr int PA = BM * TK / 4, LA = PA < THREADS ? 1 : PA / THREADS, LW = BN * TK / 4 / THREADS;
    static_assert((PA < THREADS || LA * THREADS == PA) && LW * THREADS * 4 == BN * TK, "the threads fetch whole pieces");
    static_assert(TN % 4 == 0 && (TM == 2 || TM % 4 == 0), "fragments are read 8 or 16 bytes at a time");
    extern __shared__ __align__(16) float tile_smem[];
    float *sa = tile_smem, *sw = tile_smem + 2 * TK * (BM + 4);
    pdl_sync();
    const int m0 = (int)(blockIdx.x % tiles_m) * BM, n0 = (int)(blockIdx.x / tiles_m) * BN;
    const int k_lo = blockIdx.z * k_slice, k_hi = min(K, k_lo + k_slice);
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;

    const TA *ra[LA];
    const TW *rw[LW];
    bool oka[LA], okw[LW];
    const int kc = (threadIdx.x % (TK / 4)) * 4, r0 = threadIdx.x / (TK / 4);
    constexpr int RSTEP = THREADS / (TK / 4);
#pragma unroll
    for (int i = 0; i < LA; i++) { const int r = m0 + r0 + RSTEP * i; oka[i] = r < M && r0 + RSTEP * i < BM; ra[i] = a + (size_t)(oka[i] ? r : 0) * K; }
#pragma unroll
    for (int i = 0; i < LW; i++) { const int r = n0 + r0 + RSTEP * i; okw[i] = r < N; rw[i] = w + (size_t)(okw[i] ? r : 0) * K; }
    float4 va[LA], vw[LW];
    auto fetch = [&](int k) {
#pragma unroll
        for (int i = 0; i < LA; i++) va[i] = load4<TA, VEC>(ra[i], k + kc, k_hi, oka[i]);
#pragma unroll
        for (int i = 0; i < LW; i++) vw[i] = load4<TW, VEC>(rw[i], k + kc, k_hi, okw[i]);
    };
    auto put = [&](int b) {
        float *pa = sa + b * TK * (BM + 4) + kc * (BM + 4) + r0, *pw = sw + b * TK * (BN + 4) + kc * (BN + 4) + r0;
#pragma unroll
        for (int i = 0; i < LA; i++) {
            if (PA < THREADS && r0 >= BM) break;
            pa[RSTEP * i] = va[i].x; pa[(BM + 4) + RSTEP * i] = va[i].y; pa[2 * (BM + 4) + RSTEP * i] = va[i].z; pa[3 * (BM + 4) + RSTEP * i] = va[i].w;
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            pw[RSTEP * i] = vw[i].x; pw[(BN + 4) + RSTEP * i] = vw[i].y; pw[2 * (BN + 4) + RSTEP * i] = vw[i].z; pw[3 * (BN + 4) + RSTEP * i] = vw[i].w;
        }
    };
    // a thread's rows: groups of 4 (or 2) that lie BM / groups apart, its features: groups of 4, so that the lanes of a warp
    // read neighbouring 16-byte pieces
    constexpr int GM = TM >= 4 ? 4 : TM, NGM = TM / GM, NGN = TN / 4;
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;       // two zeros

    int b = 0;
    if (k_lo < k_hi) { fetch(k_lo); put(0); }
    __syncthreads();
    for (int k0 = k_lo; k0 < k_hi; k0 += TK) {
        const bool more = k0 + TK < k_hi;
        if (more) fetch(k0 + TK);
        const float *pa = sa + b * TK * (BM + 4), *pw = sw + b * TK * (BN + 4);
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            float av[TM];
            unsigned long long wv[TN / 2];
#pragma unroll
            for (int g = 0; g < NGM; g++) {
                if constexpr (GM == 4) {
                    const float4 x = *(const float4 *)(pa + kk * (BM + 4) + g * (BM / NGM) + ty * 4);
                    av[4 * g] = x.x; av[4 * g + 1] = x.y; av[4 * g + 2] = x.z; av[4 * g + 3] = x.w;
                } else {
                    const float2 x = *(const float2 *)(pa + kk * (BM + 4) + ty * 2);
                    av[0] = x.x; av[1] = x.y;
                }
            }
#pragma unroll
            for (int g = 0; g < NGN; g++) {
                const ulonglong2 x = *(const ulonglong2 *)(pw + kk * (BN + 4) + g * (BN / NGN) + tx * 4);
                wv[2 * g] = x.x; wv[2 * g + 1] = x.y;
            }
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const unsigned long long aa = pack2(av[i], av[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; j++) fma2(acc[i][j], aa, wv[j]);
            }
        }
        if (more) put(b ^ 1);
        __syncthreads();
        b ^= 1;
    }

    auto row_of = [&](int i) { return (i / GM) * (BM / NGM) + ty * GM + i % GM; };
    auto finish = [&](int gm, int gn, float v) {
        if (gm >= M || gn >= N) return;
        if (bias) v += load_any(bias, bias_dt, gn);
        const size_t o = (size_t)gm * N + gn;
        if (accumulate) ((float *)out)[o] += v;
        else store_any(out, out_dt, o, v);
    };
    if (gridDim.z == 1) {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
                const float2 v = unpack2(acc[i][j]);
                const int gn = n0 + (j / 2) * (BN / NGN) + tx * 4 + (j & 1) * 2;
                finish(m0 + row_of(i), gn, v.x);
                finish(m0 + row_of(i), gn + 1, v.y);
            }
        return;
    }
    // the slices' sums, in the order of the slices; rows are shared out among the CTAs of the cluster
    float *sums = tile_smem;                       // (every thread is past its last read of the stages)
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) {
            const float2 v = unpack2(acc[i][j]);
            *(float2 *)(sums + row_of(i) * BN + (j / 2) * (BN / NGN) + tx * 4 + (j & 1) * 2) = v;
        }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(sums);
    const int rows_each = BM / gridDim.z, first = blockIdx.z * rows_each;
    for (int e = threadIdx.x; e < rows_each * BN; e += THREADS) {
        const int r = first + e / BN, c = e % BN;
        float v = 0.f;
        for (unsigned s = 0; s < gridDim.z; s++) {
            uint32_t at;
            float x;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine + (uint32_t)(r * BN + c) * 4u), "r"(s));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at) : "memory");
            v += x;
        }
        finish(m0 + r, n0 + c, v);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---- few rows: the weights are streamed once ---------------------------------------------------------------------------
constexpr int ROWS_MAX = 8;          // rows this form takes
constexpr int ROWS_N = 4;            // weight rows a warp has under way
constexpr int ROWS_WARPS = 8;

// Every warp its own weight rows, or (SHARED) the warps of a block the same ones and each a share of k, 128 at a time in turn.
template <typename TA, typename TW, int MR, bool SHARED, bool VEC>
__global__ void __launch_bounds__(ROWS_WARPS * 32)
linear_rows_kernel(const TA *__restrict__ a, const TW *__restrict__ w, const void *bias, int bias_dt, void *out, int out_dt,
                   int accumulate, int M, int N, int K)
{
    __shared__ float part[SHARED ? ROWS_WARPS * MR * ROWS_N : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n0 = (SHARED ? (long long)blockIdx.x : (long long)blockIdx.x * ROWS_WARPS + warp) * ROWS_N;
    pdl_sync();
    if (n0 >= N) return;                           // (SHARED: never, a block has rows)
    const TW *rw[ROWS_N];
#pragma unroll
    for (int j = 0; j < ROWS_N; j++) rw[j] = w + (size_t)min(n0 + j, (long long)N - 1) * K;
    float acc[MR][ROWS_N];
#pragma unroll
    for (int i = 0; i < MR; i++)
#pragma unroll
        for (int j = 0; j < ROWS_N; j++) acc[i][j] = 0.f;
#pragma unroll 2
    for (int k = ((SHARED ? warp * 32 : 0) + lane) * 4; k < K; k += SHARED ? 128 * ROWS_WARPS : 128) {
        float4 vw[ROWS_N];
#pragma unroll
        for (int j = 0; j < ROWS_N; j++) vw[j] = load4<TW, VEC>(rw[j], k, K, true);
#pragma unroll
        for (int i = 0; i < MR; i++) {
            const float4 va = load4<TA, VEC>(a + (size_t)min(i, M - 1) * K, k, K, true);
#pragma unroll
            for (int j = 0; j < ROWS_N; j++) {
                acc[i][j] = fmaf(va.x, vw[j].x, acc[i][j]);
                acc[i][j] = fmaf(va.y, vw[j].y, acc[i][j]);
                acc[i][j] = fmaf(va.z, vw[j].z, acc[i][j]);
                acc[i][j] = fmaf(va.w, vw[j].w, acc[i][j]);
            }
        }
    }
    auto finish = [&](int i, int j, float v) {
        if (i >= M || n0 + j >= N) return;
        if (bias) v += load_any(bias, bias_dt, n0 + j);
        const size_t o = (size_t)i * N + n0 + j;
        if (accumulate) ((float *)out)[o] += v;
        else store_any(out, out_dt, o, v);
    };
#pragma unroll
    for (int i = 0; i < MR; i++)
#pragma unroll
        for (int j = 0; j < ROWS_N; j++) {
            const float v = warp_sum(acc[i][j]);
            if (lane == i * ROWS_N + j) {
                if (SHARED) part[warp * MR * ROWS_N + lane] = v;
                else finish(i, j, v);
            }
        }
    if (SHARED) {
        __syncthreads();
        if (threadIdx.x < MR * ROWS_N) {
            float v = 0.f;
#pragma unroll
            for (int s = 0; s < ROWS_WARPS; s++) v += part[s * MR * ROWS_N + threadIdx.x];
            finish(threadIdx.x / ROWS_N, threadIdx.x % ROWS_N, v);
        }
    }
}
static_assert(ROWS_MAX * ROWS_N <= 32, "a lane stores one sum");

struct Product {
    const void *a, *w, *bias; int bias_dt; void *out; int out_dt, accumulate, M, N, K; cudaStream_t st;
};

template <typename TA, typename TW, int BM, int BN, int TM, int TN, bool VEC>
static cudaError_t launch_tile(const Product &p, int splits)
{
    constexpr size_t smem = (size_t)tile_floats<BM, BN>() * sizeof(float);
    auto kernel = linear_tile_kernel<TA, TW, BM, BN, TM, TN, VEC>;
    static bool configured[64] = {false};
    const int dev = current_device();
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    const int tiles_m = (p.M + BM - 1) / BM, tiles_n = (p.N + BN - 1) / BN;
    const int k_slice = ((p.K + splits - 1) / splits + TK - 1) / TK * TK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles_m * (unsigned)tiles_n, 1, splits);
    cfg.blockDim = dim3((BM / TM) * (BN / TN));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = p.st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = splits;
        n++;
    }
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, (const TA *)p.a, (const TW *)p.w, p.bias, p.bias_dt, p.out, p.out_dt, p.accumulate, p.M, p.N, p.K, tiles_m, k_slice);
}

// Rows of its own for every warp where that fills the SMs twice over; else the warps of a block share them: 896 features of
// 4,864 are 28 blocks one way (47 us, most SMs idle) and 224 the other (see hfb_linear_plain).
template <typename TA, typename TW, int MR, bool VEC>
static cudaError_t launch_rows(const Product &p, int sms)
{
    const long long groups = (p.N + (long long)ROWS_N - 1) / ROWS_N;
    const bool shared = groups / ROWS_WARPS < 2 * sms;
    const unsigned grid = (unsigned)(shared ? groups : (groups + ROWS_WARPS - 1) / ROWS_WARPS);
    return launch_pdl(shared ? linear_rows_kernel<TA, TW, MR, true, VEC> : linear_rows_kernel<TA, TW, MR, false, VEC>, dim3(grid), dim3(ROWS_WARPS * 32), 0, p.st,
                      (const TA *)p.a, (const TW *)p.w, p.bias, p.bias_dt, p.out, p.out_dt, p.accumulate, p.M, p.N, p.K);
}

// The shape of the many-row form: the tile (0: 128 x 128, 1: 64 x 64, 2: 16 x 64) and the slices of k with the least time
// by a count of multiply-adds on the busiest SM.  A larger tile does more per value it reads from shared memory (4,096 rows of
// 4,096 x 4,096: 54 TFLOP/s with 128 x 128, 40 with 64 x 64), a smaller one and more slices spread better (333 rows, 896 x
// 4,864: 42 tiles in 8 slices each 123 us, unsliced 487; 12 rows of the same: 41 us with 16 x 64 in 8 slices, 291 unsliced).
struct TileChoice { int tile, splits; };
static TileChoice choose_tile(int M, int N, int K, int sms)
{
    static const int bm[3] = {128, 64, 16}, bn[3] = {128, 64, 64};
    static const double rate[3] = {1.0, 0.75, 0.35};
    TileChoice best{0, 1};
    double best_cost = -1.0;
    for (int t = 0; t < 3; t++) {
        const double tiles = (double)((M + bm[t] - 1) / bm[t]) * (double)((N + bn[t] - 1) / bn[t]);
        for (int s = 1; s <= MAX_SPLITS; s *= 2) {
            if (s > 1 && K / s < 128) break;
            const double each = (double)bm[t] * bn[t] * (((K + s - 1) / s) + 48);           // 48: filling the stages, storing
            const double per_sm = tiles * s / sms, rounds = per_sm <= 1.0 ? 1.0 : per_sm < 4.0 ? (double)(long)(per_sm + 0.999) : per_sm;
            // one CTA alone on an SM leaves its units waiting for shared memory now and then
            const double cost = each * rounds / rate[t] * (per_sm <= 1.0 ? 1.25 : 1.0) * (s > 1 ? 1.05 : 1.0);
            if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best = TileChoice{t, s}; }
        }
    }
    return best;
}

static int sm_total()
{
    static int n[64] = {0};
    const int dev = current_device();
    if (!n[dev] && (cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n[dev] <= 0)) n[dev] = 1;
    return n[dev];
}

template <typename TA, typename TW, bool VEC>
static cudaError_t launch_product(const Product &p)
{
    const int sms = sm_total();
    if (p.M <= ROWS_MAX) {
        if (p.M == 1) return launch_rows<TA, TW, 1, VEC>(p, sms);
        if (p.M == 2) return launch_rows<TA, TW, 2, VEC>(p, sms);
        if (p.M <= 4) return launch_rows<TA, TW, 4, VEC>(p, sms);
        return launch_rows<TA, TW, 8, VEC>(p, sms);
    }
    const TileChoice c = choose_tile(p.M, p.N, p.K, sms);
    if (c.tile == 0) return launch_tile<TA, TW, 128, 128, 8, 8, VEC>(p, c.splits);
    if (c.tile == 1) return launch_tile<TA, TW, 64, 64, 4, 8, VEC>(p, c.splits);
    return launch_tile<TA, TW, 16, 64, 2, 4, VEC>(p, c.splits);
}

}  // namespace hfb

using namespace hfb;

extern "C" int hfb_linear_plain(const void *a, int a_dt, const void *w, int w_dt, const void *bias, int bias_dt,
                                void *out, int out_dt, int accumulate, int M, int N, int K, hfb_stream s)
{
    if (M <= 0 || N <= 0) return HFB_OK;
    if (!valid_dt(a_dt) || !valid_dt(w_dt) || !valid_dt(out_dt) || (bias && !valid_dt(bias_dt)) || K <= 0)
        return fail(HFB_EINVAL, "linear: bad arguments (M=%d N=%d K=%d)", M, N, K);
    if (accumulate && out_dt != HFB_F32) return fail(HFB_EINVAL, "linear: accumulation needs a float32 output");
    if ((M + 63) / 64 > 65535) return fail(HFB_ENOTSUP, "linear: %d rows exceed the plain kernel's grid", M);
    const Product p{a, w, bias, bias_dt, out, out_dt, accumulate, M, N, K, (cudaStream_t)s};
    // Up to 8 rows stream the weights (1 row, 151,936 x 896: 100 us = 5.4 TB/s, 289 us with tiles); from there on the tiles are
    // level with them (8 rows, 9,728 x 896: 31 us streamed, 39 tiled; 12 rows: 39 tiled) and their time hardly grows with the rows.
    // pieces of four values where every row starts on a multiple of them
    const uintptr_t am = a_dt == HFB_F32 ? 15 : 7, wm = w_dt == HFB_F32 ? 15 : 7;
    const bool vec = (K & 3) == 0 && ((uintptr_t)a & am) == 0 && ((uintptr_t)w & wm) == 0;
#define LAUNCH(TA, TW) g_launch_err = vec ? launch_product<TA, TW, true>(p) : launch_product<TA, TW, false>(p)
    if (a_dt == HFB_F32 && w_dt == HFB_F32) LAUNCH(float, float);
    else if (a_dt == HFB_F32) LAUNCH(float, __nv_bfloat16);
    else if (w_dt == HFB_F32) LAUNCH(__nv_bfloat16, float);
    else LAUNCH(__nv_bfloat16, __nv_bfloat16);
#undef LAUNCH
    return check_pdl_launch(g_launch_err, "linear_plain");
}
