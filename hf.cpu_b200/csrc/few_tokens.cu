// Products of up to eight tokens that start at the float32 stream and end where the next kernel begins: norm, product, and the sum
// with the stream, the gated pair, or rotation and cache write, in one kernel.
//
// A layer of a small model reads a few megabytes in a step of single tokens, far less than its kernels' boundaries cost.  The
// split product and the tail that sums its slices are two kernels (for the whole layer eight); here a block keeps the whole inner
// dimension of its features, so the sums are finished where they are made, and the norm in front is a factor on them: five.
// The block's rows of w are asked for before the wait for the kernel in front (they depend on nothing), so they are on their way
// to shared memory, all of them, while that kernel still runs; what is left behind the wait is one trip to L2 for x, a few products
// of mma.sync m16n8k16 (features on the columns, tokens on the rows, the warps share k) and one sum over the warps.  tcgen05 would
// bring nothing: eight tokens fill an eighth of its narrowest tile, and its accumulator's trip through TMEM is latency.
// The kernel behind is released when the wait returns: released at entry, its copies and those of the one behind it came before this
// one's (eight steps of one token, 0.5B sizes: 5.07 against 4.63 ms).
// Measured, a layer of the 0.5B sizes in a step of one token: 30 us with split products and their tails, 21 now; 896 x 896 and
// 9,728 x 896, one token, added to the stream, weights out of L2, launches overlapping: 2.3 and 6.0 us, 6.1 and 6.6 the split products.
// Every block runs at once, one an SM: the rule (few_groups) takes matrices of which an SM holds its share in shared memory.
#include "common.cuh"

static thread_local cudaError_t g_launch_err = cudaSuccess;      // what the last launch_pdl returned

namespace hfb {
int *error_word();

enum { FEW_STORE = 0, FEW_ADD = 1, FEW_GLU = 2, FEW_ROPE = 3 };

struct FewParams {
    int M, N, K;
    const __nv_bfloat16 *w;            // [N, K]
    const void *x;                     // bfloat16 [M, K]; with norm_w float32 [M, K], normed on the way in
    const void *norm_w; int norm_dt;   // [K] or null
    float eps;
    int mode;
    int act;                           // FEW_GLU: the gate's activation; FEW_STORE: 0 none, else the HFB_ACT_* code
    float glu_limit, glu_alpha, glu_offset;
    const void *bias; int bias_dt;     // [N] or null
    void *out; int out_dt;             // [M, N] ([M, N / 2] with FEW_GLU)
    long long ldo;                     // elements between rows of out
    // FEW_ROPE: the output is the q|k|v row of a token; queries go to out, keys and values to the token's cache slot
    const float *cos_sin; int n_positions;
    const int32_t *positions, *slots;
    __nv_bfloat16 *k_cache, *v_cache;
    long long cache_slots;
    int H, G, d;
};

constexpr int FEW_CHUNK = 32;          // of k a warp takes at a time
constexpr int FEW_SMEM_MAX = 200 * 1024;
constexpr int MAX_M = 8, WARPS = 8, THREADS = WARPS * 32, SS_BYTES = MAX_M * WARPS * 4;

__device__ __forceinline__ void few_mma(float (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}

// Bytes between rows in shared memory: 64 past a multiple of 128, so that two neighbouring rows' pieces of 64 bytes lie in
// different banks.
__host__ __device__ inline int few_stride(int K) { return ((K + FEW_CHUNK - 1) / FEW_CHUNK * FEW_CHUNK * 2 + 127) / 128 * 128 + 64; }

__device__ __forceinline__ float few_act(float z, int act)
{
    if (act == HFB_ACT_RELU) return fmaxf(z, 0.f);
    if (act == HFB_ACT_RELU2) { const float r = fmaxf(z, 0.f); return r * r; }
    if (act == HFB_ACT_GELU_TANH) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    return z / (1.0f + expf(-z));
}

template <int N> struct Count { static constexpr int value = N; };

// NG groups of eight features a block.
template <int NG>
__global__ void __launch_bounds__(THREADS, NG <= 8 ? 3 : 2) few_kernel(const FewParams p, int *err)
{
    extern __shared__ __align__(128) unsigned char few_sm[];
    float *ss = (float *)few_sm;                               // [MAX_M][WARPS] sums of squares
    unsigned char *sm = few_sm + SS_BYTES;
    HFB_TRACE_ENTRY(17);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int chunks = (p.K + FEW_CHUNK - 1) / FEW_CHUNK, pieces = chunks * (FEW_CHUNK / 8), stride = few_stride(p.K);
    constexpr int F = NG * 8;
    unsigned char *sx = sm + (size_t)F * stride;
    auto copy16 = [&](unsigned char *dst, const __nv_bfloat16 *src, bool in) {
        const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(to), "l"(src), "r"(in ? 16 : 0) : "memory");
    };
    for (int r = warp; r < F; r += WARPS) {
        const int j = r >> 3;
        int f;
        if (p.mode == FEW_ROPE) {                            // groups in pairs, half a head apart
            const int half = p.d >> 1, pr = ((int)blockIdx.x * NG + j) >> 1, per = half >> 3;
            f = pr / per * p.d + pr % per * 8 + (j & 1) * half + (r & 7);
        } else f = (int)blockIdx.x * F + r;
        if (f >= p.N) continue;                              // (what its place holds ends in features that are not stored)
        const __nv_bfloat16 *src = p.w + (size_t)f * p.K;
        for (int i = lane; i < pieces; i += 32) copy16(sm + (size_t)r * stride + i * 16, i * 8 < p.K ? src + i * 8 : p.w, i * 8 < p.K);
    }
    pdl_sync();
    // ---- x into shared memory; the normed form rounds x * w and leaves the row's factor to the finished sums
    const int per_row = p.M == 1 ? WARPS : p.M == 2 ? WARPS / 2 : p.M <= 4 ? WARPS / 4 : 1, part = warp % per_row;     // warps to a row
    if (!p.norm_w) {
        for (int m = warp / per_row; m < p.M; m += WARPS / per_row) {
            const __nv_bfloat16 *src = (const __nv_bfloat16 *)p.x + (size_t)m * p.K;
            for (int i = part * 32 + lane; i < pieces; i += per_row * 32) copy16(sx + (size_t)m * stride + i * 16, i * 8 < p.K ? src + i * 8 : src, i * 8 < p.K);
        }
    } else {
        // U quads of a row a lane at a time, the reads of all of them in flight
        auto norm_rows = [&](auto count) {
            constexpr int U = decltype(count)::value;
            const int quads = pieces * 2, step = per_row * 32;
            for (int m = warp / per_row; m < p.M; m += WARPS / per_row) {
                const float *xr = (const float *)p.x + (size_t)m * p.K;
                float s = 0.f;
                for (int i0 = part * 32 + lane; i0 < quads; i0 += U * step) {
                    float4 v[U], nw[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int i = i0 + u * step;
                        v[u] = nw[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (i * 4 < p.K) { v[u] = *(const float4 *)(xr + i * 4); nw[u] = load_any4(p.norm_w, p.norm_dt, i * 4); }
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int i = i0 + u * step;
                        s += v[u].x * v[u].x + v[u].y * v[u].y + v[u].z * v[u].z + v[u].w * v[u].w;
                        if (i < quads)
                            store_any4(sx + (size_t)m * stride, HFB_BF16, i * 4,
                                       make_float4(v[u].x * nw[u].x, v[u].y * nw[u].y, v[u].z * nw[u].z, v[u].w * nw[u].w));
                    }
                }
                s = warp_sum(s);
                if (lane == 0) ss[m * WARPS + part] = s;
            }
        };
        if (pieces * 2 <= per_row * 32) norm_rows(Count<1>());
        else if (pieces * 2 <= per_row * 64) norm_rows(Count<2>());
        else norm_rows(Count<8>());
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- products: a lane reads sixteen bytes of a row of each operand, the k of two products (any order of k serves)
    float acc[NG][4];
#pragma unroll
    for (int j = 0; j < NG; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const unsigned char *xa = sx + (size_t)g * stride + t * 16, *wa = sm + (size_t)g * stride + t * 16;
    const bool live = g < p.M;
    for (int c = warp; c < chunks; c += WARPS) {
        const uint4 a = live ? *(const uint4 *)(xa + c * (FEW_CHUNK * 2)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int j = 0; j < NG; j++) {
            const uint4 b = *(const uint4 *)(wa + (size_t)j * 8 * stride + c * (FEW_CHUNK * 2));
            few_mma(acc[j], a.x, a.y, b.x, b.y);
            few_mma(acc[j], a.z, a.w, b.z, b.w);
        }
    }
    // ---- the warps' sums meet where the weights were: red[warp][token][features]
    __syncthreads();
    float *red = (float *)sm;
#pragma unroll
    for (int j = 0; j < NG; j++)
        if (live) *(float2 *)(red + ((size_t)warp * p.M + g) * F + j * 8 + 2 * t) = make_float2(acc[j][0], acc[j][1]);
    __syncthreads();
    auto sum = [&](int m, int f) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) v += red[((size_t)w * p.M + m) * F + f];
        return v;
    };
    auto scale = [&](int m) {
        if (!p.norm_w) return 1.f;
        float s = 0.f;
        for (int i = 0; i < per_row; i++) s += ss[m * WARPS + i];
        return 1.0f / sqrtf(s / (float)p.K + p.eps);
    };
    const int base = blockIdx.x * F;
    if (p.mode == FEW_GLU) {
        for (int i = threadIdx.x; i < p.M * (F / 2); i += THREADS) {
            const int m = i / (F / 2), h = i - m * (F / 2), f = base + 2 * h;
            if (f >= p.N) continue;
            const float r = scale(m);
            float gt = sum(m, 2 * h) * r, up = sum(m, 2 * h + 1) * r;
            if (p.bias) { gt += load_any(p.bias, p.bias_dt, f); up += load_any(p.bias, p.bias_dt, f + 1); }
            float v;
            if (p.act == HFB_ACT_CLAMPED_GLU) {
                gt = fminf(gt, p.glu_limit);
                up = fminf(fmaxf(up, -p.glu_limit), p.glu_limit);
                v = __fdividef(gt, 1.0f + __expf(-p.glu_alpha * gt)) * (up + p.glu_offset);
            } else v = few_act(gt, p.act) * up;
            store_any(p.out, p.out_dt, (size_t)m * p.ldo + (f >> 1), v);
        }
    } else if (p.mode == FEW_ROPE) {
        constexpr int P = NG / 2 > 0 ? NG / 2 * 8 : 8;
        const int half = p.d >> 1, per = half >> 3;
        for (int i = threadIdx.x; i < p.M * P; i += THREADS) {
            const int m = i / P, h = i - m * P, j = h >> 3, e = h & 7;
            const int pr = (int)blockIdx.x * (NG / 2) + j, head = pr / per, in = pr % per * 8 + e, f = head * p.d + in;
            if (f >= p.N) continue;
            const float r = scale(m);
            float a = sum(m, j * 16 + e) * r, b = sum(m, j * 16 + 8 + e) * r;
            if (p.bias) { a += load_any(p.bias, p.bias_dt, f); b += load_any(p.bias, p.bias_dt, f + half); }
            __nv_bfloat16 *dst;
            if (head < p.H) dst = (__nv_bfloat16 *)p.out + (size_t)m * p.H * p.d + f;
            else {
                long long slot = p.slots ? p.slots[m] : -1;
                if (slot >= p.cache_slots) { atomicOr(err, HFB_ERR_SLOT); slot = -1; }
                if (slot < 0) continue;
                dst = (head < p.H + p.G ? p.k_cache + ((size_t)slot * p.G + (head - p.H)) * p.d
                                        : p.v_cache + ((size_t)slot * p.G + (head - p.H - p.G)) * p.d) + in;
            }
            if (head < p.H + p.G) {
                int pos = p.positions[m];
                if (pos < 0 || pos >= p.n_positions) { atomicOr(err, HFB_ERR_POSITION); pos = 0; }
                const float2 cs = *(const float2 *)(p.cos_sin + ((size_t)pos * half + in) * 2);
                float lo, hi;
                rope_pair(to_f32(__float2bfloat16_rn(a)), to_f32(__float2bfloat16_rn(b)), cs.x, cs.y, lo, hi);
                a = lo; b = hi;
            }
            dst[0] = __float2bfloat16_rn(a);
            dst[half] = __float2bfloat16_rn(b);
        }
    } else {
        for (int i = threadIdx.x; i < p.M * F; i += THREADS) {
            const int m = i / F, h = i - m * F, f = base + h;
            if (f >= p.N) continue;
            float v = sum(m, h) * scale(m);
            if (p.bias) v += load_any(p.bias, p.bias_dt, f);
            if (p.mode == FEW_ADD) ((float *)p.out)[(size_t)m * p.ldo + f] += v;
            else store_any(p.out, p.out_dt, (size_t)m * p.ldo + f, p.act ? few_act(v, p.act) : v);
        }
    }
}

static size_t few_smem(int M, int K, int NG)
{
    const size_t rows = (size_t)(NG * 8 + M) * few_stride(K), sums = (size_t)WARPS * M * NG * 8 * 4;
    return SS_BYTES + (rows > sums ? rows : sums);
}

template <int NG>
static int launch_few(const FewParams &p, cudaStream_t st)
{
    static bool configured[64] = {false};
    const int dev = current_device();
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(few_kernel<NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_SMEM_MAX);
        if (e != cudaSuccess) return fail(HFB_ECUDA, "few_tokens: cannot opt in to shared memory: %s", cudaGetErrorString(e));
        configured[dev] = true;
    }
    const int groups = (p.N + 7) / 8;
    g_launch_err = launch_pdl(few_kernel<NG>, dim3((groups + NG - 1) / NG), dim3(THREADS), few_smem(p.M, p.K, NG), st, p, error_word());
    return check_pdl_launch(g_launch_err, "few_tokens");
}

static int few_sms()
{
    static int n[64] = {0};
    const int dev = current_device();
    if (!n[dev] && (cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n[dev] <= 0)) n[dev] = 1;
    return n[dev];
}

// Groups of eight features a block, so that the blocks run at once, one an SM (0: no block holds that many rows).
static int few_groups(int M, int N, int K, bool pairs)
{
    const int each = ((N + 7) / 8 + few_sms() - 1) / few_sms(), sizes[] = {1, 2, 3, 4, 5, 6, 8, 10, 12};
    for (int ng : sizes)
        if (ng >= each && !(pairs && (ng & 1))) return few_smem(M, K, ng) <= FEW_SMEM_MAX ? ng : 0;
    return 0;
}

// (sizes that no share fits are turned down before the arithmetic on them, which is in 32 bits)
static bool few_takes(int M, int N, int K, bool pairs)
{
    return M >= 1 && M <= MAX_M && K >= 8 && (K & 7) == 0 && K <= FEW_SMEM_MAX && N >= 8 && N <= (1 << 30) && few_groups(M, N, K, pairs) > 0;
}

static int few_launch(const FewParams &p, cudaStream_t st)
{
    switch (few_groups(p.M, p.N, p.K, p.mode == FEW_ROPE)) {
    case 1: return launch_few<1>(p, st);
    case 2: return launch_few<2>(p, st);
    case 3: return launch_few<3>(p, st);
    case 4: return launch_few<4>(p, st);
    case 5: return launch_few<5>(p, st);
    case 6: return launch_few<6>(p, st);
    case 8: return launch_few<8>(p, st);
    case 10: return launch_few<10>(p, st);
    default: return launch_few<12>(p, st);
    }
}

}  // namespace hfb

using namespace hfb;

static int few_fill(const char *who, FewParams &p, const void *x, const void *norm_w, int norm_dt, float eps, const void *w, const void *bias, int bias_dt, int M, int N, int K)
{
    if (!few_takes(M, N, K, p.mode == FEW_ROPE)) return fail(HFB_ENOTSUP, "%s: M=%d N=%d K=%d is not a product of few tokens", who, M, N, K);
    if ((norm_w && !valid_dt(norm_dt)) || (bias && !valid_dt(bias_dt))) return fail(HFB_EINVAL, "%s: bad element types", who);
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || (norm_w && !aligned4(norm_w, norm_dt))) return fail(HFB_ENOTSUP, "%s: operands must be 16-byte aligned", who);
    p.M = M; p.N = N; p.K = K; p.x = x; p.norm_w = norm_w; p.norm_dt = norm_dt; p.eps = eps; p.w = (const __nv_bfloat16 *)w;
    p.bias = bias; p.bias_dt = bias_dt; p.ldo = N;
    return HFB_OK;
}

extern "C" int hfb_few_takes(int M, int N, int K, int rope) { return few_takes(M, N, K, rope != 0) ? 1 : 0; }

extern "C" int hfb_few_linear(const void *x, const void *norm_w, int norm_dt, float eps, const void *w, const void *bias, int bias_dt, void *out, int out_dt,
                              int accumulate, int act, int M, int N, int K, hfb_stream s)
{
    if (M <= 0 || N <= 0) return HFB_OK;
    FewParams p{};
    const int rc = few_fill("few_linear", p, x, norm_w, norm_dt, eps, w, bias, bias_dt, M, N, K);
    if (rc != HFB_OK) return rc;
    if (!valid_dt(out_dt) || (accumulate && (out_dt != HFB_F32 || act)) || act < 0 || act >= HFB_ACT_NONE)
        return fail(HFB_EINVAL, "few_linear: accumulation needs a float32 output and no activation");
    p.act = act;
    p.mode = accumulate ? FEW_ADD : FEW_STORE; p.out = out; p.out_dt = out_dt;
    return few_launch(p, (cudaStream_t)s);
}

extern "C" int hfb_few_glu(const void *x, const void *norm_w, int norm_dt, float eps, const void *w, const void *bias, int bias_dt, void *out, int out_dt,
                           int64_t ldo, int M, int N, int K, int act, float limit, float alpha, float offset, hfb_stream s)
{
    if (M <= 0 || N <= 0) return HFB_OK;
    FewParams p{};
    const int rc = few_fill("few_glu", p, x, norm_w, norm_dt, eps, w, bias, bias_dt, M, N, K);
    if (rc != HFB_OK) return rc;
    if ((N & 1) || !valid_dt(out_dt) || act < 0 || (act >= HFB_ACT_NONE && act != HFB_ACT_CLAMPED_GLU) || (ldo && ldo < N / 2))
        return fail(HFB_EINVAL, "few_glu: bad arguments");
    p.mode = FEW_GLU; p.act = act; p.glu_limit = limit; p.glu_alpha = alpha; p.glu_offset = offset; p.out = out; p.out_dt = out_dt; p.ldo = ldo ? ldo : N / 2;
    return few_launch(p, (cudaStream_t)s);
}

extern "C" int hfb_few_rope_kv(const void *x, const void *norm_w, int norm_dt, float eps, const void *w, const void *bias, int bias_dt, const float *cos_sin,
                               int n_positions, const int32_t *positions, const int32_t *slots, void *q_out, void *k_cache, void *v_cache,
                               int64_t cache_slots, int M, int K, int H, int G, int d, hfb_stream s)
{
    if (M <= 0) return HFB_OK;
    if ((d != 64 && d != 128) || H <= 0 || G <= 0 || !cos_sin || !positions || n_positions <= 0 || ((uintptr_t)cos_sin & 7))
        return fail(HFB_ENOTSUP, "few_rope_kv: takes head sizes 64 and 128 and a rotation table");
    FewParams p{};
    p.mode = FEW_ROPE;
    const int rc = few_fill("few_rope_kv", p, x, norm_w, norm_dt, eps, w, bias, bias_dt, M, (H + 2 * G) * d, K);
    if (rc != HFB_OK) return rc;
    p.out = q_out; p.out_dt = HFB_BF16; p.cos_sin = cos_sin; p.n_positions = n_positions; p.positions = positions; p.slots = slots;
    p.k_cache = (__nv_bfloat16 *)k_cache; p.v_cache = (__nv_bfloat16 *)v_cache; p.cache_slots = cache_slots; p.H = H; p.G = G; p.d = d;
    return few_launch(p, (cudaStream_t)s);
}
