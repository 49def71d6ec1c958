// out[M,N] (=|+=) a[M,K] . w[N,K]^T (+ bias): the plain matrix product.
//
// Float32 multiply-adds only, any sizes, any mix of float32 / bfloat16 operands.  It is the whole float32 path's product and
// the comparison for the tensor-core kernels, in the way the reference keeps portable kernels beside its vector ones
// (src/kern_generic.c:84-91 beside src/kern_avx2.c:79-95; call shape src/model.c:419-425).
//
// An output element has ONE order of summation, whatever number of rows the product has: k is cut into slices whose number and
// length depend on N and K alone (k_slices), the products of a slice are added one by one in ascending k, and the slices' sums
// are added in their order.  So a token's float32 results are the same bits in a step of single tokens, in a portion of a prompt
// and in any company.  The two kernels below are two ways through that order.
//
// Up to ROWS_MAX rows (single tokens) the product only streams the weights: a lane owns a slice of a weight row, whose values come
// through shared memory by cp.async in pieces of 128 bytes, many pieces ahead, and the lanes that hold a row's slices add them
// at the end.  More rows are bound by the float32 units: tiles of registers over double-buffered shared memory, the next
// piece of k on its way from global memory while one is multiplied, two neighbouring features an instruction (fma.rn.f32x2:
// each half rounds as an fma of its own, and the units stay fed while other instructions issue).  A CTA walks all the slices
// and puts its sums onto the tile's totals in shared memory after each of them, or, where the tiles are fewer than the SMs, the
// CTAs of a cluster take a slice each and add up shares of the tile's rows over the cluster's shared memories: no workspace, no
// second pass over memory.
// Measured (B200, float32): see the rules in hfb_linear_plain and choose_tile.
#include "common.cuh"

static thread_local cudaError_t g_launch_err = cudaSuccess;      // what the last launch of this thread returned

namespace hfb {

// ---- many rows: tiles of BM x BN, TM x TN a thread -------------------------------------------------------------------
constexpr int TK = 16;               // of k a stage
constexpr int MAX_SPLITS = 8;        // CTAs of a cluster

// Four consecutive values p, those of a row from k on; zeros from K on.  VEC: K is a multiple of 4 and the rows are aligned to four values.
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T *p, int k, int K, bool live)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!live) return v;
    if (VEC) {
        if (k < K) {
            if constexpr (sizeof(T) == 4) {
                v = *(const float4 *)p;
            } else {
                const uint2 u = *(const uint2 *)p;
                const float2 lo = __bfloat1622float2(*(const __nv_bfloat162 *)&u.x), hi = __bfloat1622float2(*(const __nv_bfloat162 *)&u.y);
                v = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
    } else {
        if (k < K) v.x = to_f32(p[0]);
        if (k + 1 < K) v.y = to_f32(p[1]);
        if (k + 2 < K) v.z = to_f32(p[2]);
        if (k + 3 < K) v.w = to_f32(p[3]);
    }
    return v;
}

// Shared memory of a tile in floats: the two stages; behind them the totals of a CTA that walks several slices, in their place
// the sums of a CTA whose cluster shares the slices.
template <int BM, int BN> constexpr int stage_floats() { return 2 * TK * (BM + 4 + BN + 4); }
template <int BM, int BN> constexpr int tile_floats(bool totals)
{
    return totals ? stage_floats<BM, BN>() + BM * BN : stage_floats<BM, BN>() > BM * BN ? stage_floats<BM, BN>() : BM * BN;
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
    const int k_lo = blockIdx.z * k_slice, k_hi = gridDim.z > 1 ? min(K, k_lo + k_slice) : K;
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;

    const int kc = (threadIdx.x % (TK / 4)) * 4, r0 = threadIdx.x / (TK / 4);
    constexpr int RSTEP = THREADS / (TK / 4);
    const TA *ra = a + (size_t)(m0 + r0) * K + kc;               // (rows that do not exist are not read)
    const TW *rw = w + (size_t)(n0 + r0) * K + kc;
    const int live_a = min(M - m0, BM) - r0, live_w = N - n0 - r0;
    float4 va[LA], vw[LW];
    auto fetch = [&](int k) {
#pragma unroll
        for (int i = 0; i < LA; i++) va[i] = load4<TA, VEC>(ra + (size_t)(RSTEP * i) * K + k, k + kc, k_hi, RSTEP * i < live_a);
#pragma unroll
        for (int i = 0; i < LW; i++) vw[i] = load4<TW, VEC>(rw + (size_t)(RSTEP * i) * K + k, k + kc, k_hi, RSTEP * i < live_w);
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
    f32pair acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;       // two zeros

    // totals of the slices behind a CTA, a piece of four for every thread in turn; `next`: where the slice under way ends (a slice
    // is a whole number of stages)
    float4 *totals = (float4 *)(tile_smem + stage_floats<BM, BN>());
    int b = 0, k0 = k_lo, next = k_lo + k_slice;
    if (k_lo < k_hi) { fetch(k_lo); put(0); }
    __syncthreads();
    for (;;) {
        for (const int end = min(next, k_hi); k0 < end; k0 += TK) {
            const bool more = k0 + TK < k_hi;
            if (more) fetch(k0 + TK);
            const float *pa = sa + b * TK * (BM + 4), *pw = sw + b * TK * (BN + 4);
#pragma unroll
            for (int kk = 0; kk < TK; kk++) {
                float av[TM];
                f32pair wv[TN / 2];
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
                    const f32pair aa = pair_of(av[i], av[i]);
#pragma unroll
                    for (int j = 0; j < TN / 2; j++) acc[i][j] = fma2(aa, wv[j], acc[i][j]);
                }
            }
            if (more) put(b ^ 1);
            __syncthreads();
            b ^= 1;
        }
        if (k0 >= k_hi) break;
        const bool first = next == k_slice;
        next += k_slice;
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j += 2) {
                const float2 x = halves(acc[i][j]), y = halves(acc[i][j + 1]);
                float4 *t = totals + (i * (TN / 4) + j / 2) * THREADS + threadIdx.x;
                float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *t;
                v.x += x.x; v.y += x.y; v.z += y.x; v.w += y.y;
                *t = v;
                acc[i][j] = acc[i][j + 1] = 0ull;
            }
    }
    if (gridDim.z == 1 && next > k_slice) {                      // the last slice's sums onto the others'
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j += 2) {
                const float4 v = totals[(i * (TN / 4) + j / 2) * THREADS + threadIdx.x];
                const float2 x = halves(acc[i][j]), y = halves(acc[i][j + 1]);
                acc[i][j] = pair_of(v.x + x.x, v.y + x.y);
                acc[i][j + 1] = pair_of(v.z + y.x, v.w + y.y);
            }
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
                const float2 v = halves(acc[i][j]);
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
            const float2 v = halves(acc[i][j]);
            *(float2 *)(sums + row_of(i) * BN + (j / 2) * (BN / NGN) + tx * 4 + (j & 1) * 2) = v;
        }
    cluster_barrier();
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(sums);
    const int rows_each = BM / gridDim.z, first = blockIdx.z * rows_each;
    for (int e = threadIdx.x; e < rows_each * BN; e += THREADS) {
        const int r = first + e / BN, c = e % BN;
        float v = 0.f;
        for (unsigned s = 0; s < gridDim.z; s++) {
            const uint32_t at = map_to_rank(mine + (uint32_t)(r * BN + c) * 4u, s);
            float x;
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at) : "memory");
            v += x;
        }
        finish(m0 + r, n0 + c, v);
    }
    cluster_barrier();
}

// ---- few rows: the weights are streamed once ---------------------------------------------------------------------------
constexpr int ROWS_MAX = 8;          // rows this form takes
constexpr int PK = 32;               // values of a slice of a row that a stage holds
constexpr int ROW_THREADS = 128;
// stages of a block with ST slices of rows: three blocks an SM, or as much on its way where there is one
template <int ST> constexpr int row_stages() { return ST == 128 ? 3 : 8; }
template <typename T> constexpr int pitch() { return PK * (int)sizeof(T) + 16; }       // sixteen bytes a lane from different banks

template <int BYTES> __device__ __forceinline__ void cp_async(void *dst, const void *src, bool live)
{
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    const int size = live ? BYTES : 0;                           // (the rest is filled with zeros)
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(size) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(to), "l"(src), "n"(BYTES), "r"(size) : "memory");
}

// N values to shared memory, zeros where there are none (single bfloat16 values, which cp.async does not take, by way of a register)
template <int N, typename T> __device__ __forceinline__ void copy_values(T *dst, const T *src, bool live)
{
    if constexpr (N * sizeof(T) >= 4) cp_async<N * (int)sizeof(T)>(dst, src, live);
    else *dst = live ? *src : T(0.f);
}

// eight values of shared memory as floats
__device__ __forceinline__ void read8(const float *p, float (&x)[8])
{
    const float4 u = *(const float4 *)p, v = *(const float4 *)(p + 4);
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
}
__device__ __forceinline__ void read8(const __nv_bfloat16 *p, float (&x)[8])
{
    const uint4 v = *(const uint4 *)p;
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 f = __bfloat1622float2(*(const __nv_bfloat162 *)&u[i]);
        x[2 * i] = f.x; x[2 * i + 1] = f.y;
    }
}

// A thread is a slice of one weight row: thread = slice * rows + row.  All threads of a block bring the next stages of its ST
// slices, neighbours the parts of one piece, and the piece of the activations that belongs to it; where there are few slices of rows
// in all (ST < ROW_THREADS) most threads do nothing else.  Memory is what bounds the large products, the latencies of a stage (the
// wait, the reads of shared memory, 32 dependent multiply-adds a row) the small ones.
// Measured (B200, float32, weights from memory), 1 / 8 rows: 151,936 x 896 97 / 122 us (5.6 TB/s), 9,728 x 896 9.6 / 14.3, 896 x
// 4,864 8.3 / 18.2, 896 x 896 3.1 / 5.1.  (Lanes that share a row's k and meet in a tree: 83 / 226, 10.2 / 22, 5.9 / 12, 1.8 / 4.3
// us, but no tile adds in that order, and a token's bits would depend on how many others share its step.  Six stages of 64 slices
// and blocks that only fill an SM twice: 105 / 184 us for the first of these.)
template <typename TA, typename TW, int MR, int ST, bool VEC>
__global__ void __launch_bounds__(ROW_THREADS)
linear_rows_kernel(const TA *__restrict__ a, const TW *__restrict__ w, const void *bias, int bias_dt, void *out, int out_dt,
                   int accumulate, int M, int N, int K, int slices, int k_slice)
{
    constexpr int T = ROW_THREADS, STAGES = row_stages<ST>(), W_BYTES = ST * pitch<TW>();
    constexpr int CV = VEC ? 4 : 1, PARTS = PK / CV;             // values of a copy, copies of a piece
    constexpr int WC = ST * PARTS / T, AC = (MR * MAX_SPLITS * PARTS + T - 1) / T;       // copies of a thread
    extern __shared__ __align__(16) uint8_t ring[];
    const int t = threadIdx.x, s_log = __ffs(slices) - 1, rows = ST >> s_log, r_log = __ffs(rows) - 1;      // (powers of two)
    const int stage_bytes = W_BYTES + MR * slices * pitch<TA>();
    const long long n0 = (long long)blockIdx.x * rows;
    const int pieces = (min(k_slice, K) + PK - 1) / PK;
    // where a thread's copies come from, how many values their slices have from there on, and where they go in a stage
    const int part = t % PARTS * CV;
    const TW *w_src[WC];
    const TA *a_src[AC];
    int w_left[WC], a_left[AC];
#pragma unroll
    for (int i = 0; i < WC; i++) {
        const int s = i * (T / PARTS) + t / PARTS, at = (s >> r_log) * k_slice + part;
        const long long n = n0 + (s & (rows - 1));
        w_left[i] = n < N ? min(K - at, k_slice - part) : 0;
        w_src[i] = w + (w_left[i] > 0 ? (size_t)n * K + at : 0);
    }
#pragma unroll
    for (int i = 0; i < AC; i++) {
        const int s = i * (T / PARTS) + t / PARTS, at = (s & (slices - 1)) * k_slice + part, m = s >> s_log;
        a_left[i] = m < M ? min(K - at, k_slice - part) : 0;
        a_src[i] = a + (a_left[i] > 0 ? (size_t)m * K + at : 0);
    }
    uint8_t *const w_to = ring + t / PARTS * pitch<TW>() + part * (int)sizeof(TW), *const a_to = ring + W_BYTES + t / PARTS * pitch<TA>() + part * (int)sizeof(TA);
    pdl_sync();
    auto fetch = [&](int st) {                                   // the next piece of all slices
#pragma unroll
        for (int i = 0; i < WC; i++) {
            copy_values<CV>((TW *)(w_to + st * stage_bytes + i * (T / PARTS * pitch<TW>())), w_left[i] > 0 ? w_src[i] : w, w_left[i] > 0);
            w_src[i] += PK;
            w_left[i] -= PK;
        }
#pragma unroll
        for (int i = 0; i < AC; i++) {
            if (i * (T / PARTS) + t / PARTS >= M << s_log) break;
            copy_values<CV>((TA *)(a_to + st * stage_bytes + i * (T / PARTS * pitch<TA>())), a_left[i] > 0 ? a_src[i] : a, a_left[i] > 0);
            a_src[i] += PK;
            a_left[i] -= PK;
        }
    };
    for (int p = 0; p < STAGES - 1; p++) {
        if (p < pieces) fetch(p);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[MR];
#pragma unroll
    for (int i = 0; i < MR; i++) acc[i] = 0.f;
    const uint8_t *const mine = ring + t * pitch<TW>(), *const act = ring + W_BYTES + (t >> r_log) * pitch<TA>();
    int st = 0;
    for (int p = 0; p < pieces; p++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                         // the piece is there, and every thread is past the one before
        if (t < ST) {
#pragma unroll
            for (int q = 0; q < PK; q += 8) {
                float x[8];
                read8((const TW *)(mine + st * stage_bytes) + q, x);
#pragma unroll
                for (int i = 0; i < MR; i++) {
                    float y[8];
                    read8((const TA *)(act + st * stage_bytes + (min(i, M - 1) << s_log) * pitch<TA>()) + q, y);
#pragma unroll
                    for (int e = 0; e < 8; e++) acc[i] = fmaf(y[e], x[e], acc[i]);
                }
            }
        }
        const int to = st == 0 ? STAGES - 1 : st - 1;
        if (p + STAGES - 1 < pieces) fetch(to);
        asm volatile("cp.async.commit_group;" ::: "memory");
        st = st + 1 == STAGES ? 0 : st + 1;
    }
    // the slices' sums in their order, a thread for every row
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float *sums = (float *)ring;
#pragma unroll
    for (int i = 0; i < MR; i++)
        if (t < ST) sums[i * ST + t] = acc[i];
    __syncthreads();
    for (int e = t; e < M * rows; e += T) {
        const int i = e >> r_log, r = e & (rows - 1);
        if (n0 + r >= N) continue;
        float v = 0.f;
        for (int s = 0; s < slices; s++) v += sums[i * ST + s * rows + r];
        if (bias) v += load_any(bias, bias_dt, n0 + r);
        const size_t o = (size_t)i * N + n0 + r;
        if (accumulate) ((float *)out)[o] += v;
        else store_any(out, out_dt, o, v);
    }
}

struct Product {
    const void *a, *w, *bias; int bias_dt; void *out; int out_dt, accumulate, M, N, K; cudaStream_t st;
    int slices, k_slice;
};

template <typename TA, typename TW, int BM, int BN, int TM, int TN, bool VEC>
static cudaError_t launch_tile(const Product &p, int splits)
{
    constexpr size_t most = (size_t)tile_floats<BM, BN>(true) * sizeof(float);
    const size_t smem = (size_t)tile_floats<BM, BN>(splits < p.slices) * sizeof(float);
    auto kernel = linear_tile_kernel<TA, TW, BM, BN, TM, TN, VEC>;
    static bool configured[64] = {false};
    const int dev = current_device();
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    const int tiles_m = (p.M + BM - 1) / BM, tiles_n = (p.N + BN - 1) / BN;
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
    return cudaLaunchKernelEx(&cfg, kernel, (const TA *)p.a, (const TW *)p.w, p.bias, p.bias_dt, p.out, p.out_dt, p.accumulate, p.M, p.N, p.K, tiles_m, p.k_slice);
}

template <typename TA, typename TW, int MR, int ST, bool VEC>
static cudaError_t launch_rows_of(const Product &p)
{
    const auto bytes = [](int slices) { return row_stages<ST>() * (ST * pitch<TW>() + MR * slices * pitch<TA>()); };
    auto kernel = linear_rows_kernel<TA, TW, MR, ST, VEC>;
    static bool configured[64] = {false};
    const int dev = current_device();
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes(MAX_SPLITS));
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    const unsigned rows = ST / p.slices, grid = ((unsigned)p.N + rows - 1) / rows;
    return launch_pdl(kernel, dim3(grid), dim3(ROW_THREADS), (size_t)bytes(p.slices), p.st, (const TA *)p.a, (const TW *)p.w, p.bias, p.bias_dt, p.out,
                      p.out_dt, p.accumulate, p.M, p.N, p.K, p.slices, p.k_slice);
}

// As many slices of rows a block as threads where such blocks come near to one an SM, else a quarter as many (1 / 8 rows, 2,048 x
// 5,464: 14.8 / 19 us with 128, 14.8 / 41 with 32; 896 x 4,864: 12 / 22 with 128, 8.3 / 18 with 32).
template <typename TA, typename TW, int MR, bool VEC>
static cudaError_t launch_rows(const Product &p, int sms)
{
    return (long long)p.N * p.slices >= 96ll * sms ? launch_rows_of<TA, TW, MR, 128, VEC>(p) : launch_rows_of<TA, TW, MR, 32, VEC>(p);
}

// The slices of k of a product with N features: two, four or eight where that keeps them at 64 values and more, as long as the
// streaming form has fewer than eight warps an SM of a B200 without.  Nothing else may enter here: the rows, the device and the
// types must not change the order of a sum.  (At 128 values and more 896 x 896 would have four: 1 row 4.9 us instead of 3.1, 9 rows
// 10.1 instead of 5.8, 4,096 rows 170 instead of 186.)
static int k_slices(int N, int K, int *k_slice)
{
    int s = 1;
    while (s < MAX_SPLITS && K / (2 * s) >= 64 && (long long)N * s < 148 * 8 * 32) s *= 2;
    *k_slice = ((K + s - 1) / s + TK - 1) / TK * TK;
    return s;
}

// The shape of the many-row form: the tile (0: 128 x 128, 1: 64 x 64, 2: 16 x 64), and whether a cluster shares the slices of k
// or a CTA takes them all: the least time by a count of multiply-adds on the busiest SM.  A larger tile does more per value it
// reads from shared memory (4,096 rows of 4,096 x 4,096: 2.71 ms = 51 TFLOP/s with 128 x 128 and all slices a CTA, 3.1 ms with a
// slice a CTA, 3.5 and 3.6 ms with 64 x 64), a smaller one and a slice a CTA spread better (333 rows, 896 x 4,864: 84 tiles of 64 x
// 64 with a slice a CTA 118 us, all slices 300; 12 rows of the same: 32 us with 16 x 64, all slices 261).
struct TileChoice { int tile, splits; };
static TileChoice choose_tile(int M, int N, int K, int slices, int sms)
{
    static const int bm[3] = {128, 64, 16}, bn[3] = {128, 64, 64};
    static const double rate[3] = {1.0, 0.75, 0.35};
    TileChoice best{0, 1};
    double best_cost = -1.0;
    for (int t = 0; t < 3; t++) {
        const double tiles = (double)((M + bm[t] - 1) / bm[t]) * (double)((N + bn[t] - 1) / bn[t]);
        for (int s = 1; s <= slices; s = s < slices ? slices : slices + 1) {
            // 48: filling the stages, storing; 8: putting a slice's sums onto the totals
            const double each = (double)bm[t] * bn[t] * (((K + s - 1) / s) + 48 + (s < slices ? 8 * slices : 0));
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
        if (p.M <= 4) return launch_rows<TA, TW, 4, VEC>(p, sms);
        return launch_rows<TA, TW, 8, VEC>(p, sms);
    }
    const TileChoice c = choose_tile(p.M, p.N, p.K, p.slices, sms);
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
    if (M > 64 * 65535) return fail(HFB_ENOTSUP, "linear: %d rows are more than the plain product takes", M);
    int k_slice;
    const int slices = k_slices(N, K, &k_slice);
    const Product p{a, w, bias, bias_dt, out, out_dt, accumulate, M, N, K, (cudaStream_t)s, slices, k_slice};
    // Up to 8 rows stream the weights (8 rows, 9,728 x 896: 14.3 us, 32 in tiles; 3,584 x 3,584: 21, 38 in tiles), more take tiles,
    // whose time hardly grows up to 16 rows.  Copies of four values where every row starts on a multiple of them.
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
