// Attention over the paged cache, plain kernel: one block per (token, head).
//
// For token t at position pos of its request, head h reads key/value head h / (H/G) over keys
// lo..pos; score = dot(q, k) * scale (scale after the dot), softmax in float32, out = sum p_j v_j
// (src/model.c:499-528, src/mathx.c:77-86).  The eight warps take the keys from lo on in turn, a few neighbouring ones at a
// time (KEYS: eight up to head sizes of 128), with a running maximum and sum; their partial results are merged in a fixed
// order, so the result depends only on (lo, pos) and the values, never on what else is in the batch.
// A step over the keys is a chain of latencies (page, key, reduction over the lanes, exponential, value), so a warp asks
// for the keys and the values of a whole group at once, reduces the group's dot products together (9 exchanges between
// lanes for eight keys instead of 40) and rescales its sums once a group.  Float32, 14 heads
// of 64, 24 layers, a prompt of 333 tokens and four single tokens behind it: 18.5 -> 3.9 ms over the 120 launches.  Value heads may have another size (dv)
// than query/key heads (d): the output row of a head has dv elements.  Consecutive value rows lie v_row elements apart:
// dv for an array of values, d when the values are the first dv elements of the keys themselves (one latent row per
// token that serves as key and, without its last elements, as value).
//
// Two options of the softmax: a sink per head, a score without key or value that joins the denominator once
// (p_j = exp(s_j) / (exp(sink) + sum exp(s_j)); `sinks` [H] float32, learned, or `zero_sink` for a sink of score 0,
// which adds one to the denominator), and a bias linear in the distance, s_j -= slopes[h] * (pos - j).
// Two options of the score: a factor per head, s_j *= head_scales[h], and a cap, s_j <- softcap * tanh(s_j / softcap)
// (after the factors, before the bias and the softmax; softcap <= 0: none).
#include "common.cuh"

static thread_local cudaError_t g_launch_err = cudaSuccess;      // what the last launch_pdl returned

namespace hfb {
int *error_word();

constexpr int ATT_WARPS = 8;
constexpr int MAX_D_PER_LANE = 20;     // head sizes up to 640

// Keys a warp takes at a time, for PER_LANE elements of a head a lane (the keys and values of a group are held in registers).
template <int PER_LANE> constexpr int group_keys() { return PER_LANE <= 4 ? 8 : PER_LANE <= 8 ? 4 : 2; }

// Sums v[i] over the lanes for all N (a power of two) values at once; afterwards lane l holds the sum of value key_of<N>(l).
template <int N> __device__ __forceinline__ float group_sum(float (&v)[N])
{
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = N / 2; n > 0; n >>= 1, o >>= 1) {
        const bool high = lane & o;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float keep = high ? v[i + n] : v[i], give = high ? v[i] : v[i + n];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    float r = v[0];
    for (; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}
// (the first value lies in the lanes' upper half or not, and so on down; lane_of names one of the lanes that hold value i)
template <int N> __device__ __forceinline__ int key_of(int lane) { return lane / (32 / N); }
template <int N> __device__ __forceinline__ int lane_of(int i) { return i * (32 / N); }

template <typename T, int PER_LANE>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_plain_kernel(const T *q, const T *k_cache, const T *v_cache, const int32_t *block_table, int max_blocks,
                       const int32_t *token_seq, const int32_t *positions, int block_size, long long num_pages,
                       int window, float scale, T *out, int H, int G, int d, int dv, int v_row, const float *sinks, int zero_sink,
                       const float *slopes, const float *head_scales, float softcap, int *err)
{
    constexpr int KEYS = group_keys<PER_LANE>();
    pdl_sync();
    int t = blockIdx.x, h = blockIdx.y;
    int g = h / (H / G);
    int seq = token_seq[t], pos = positions[t];
    int lo = mask_lo(pos, window);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t *table = block_table + (size_t)seq * max_blocks;

    __shared__ float s_m[ATT_WARPS], s_l[ATT_WARPS];
    __shared__ float s_acc[ATT_WARPS][32 * PER_LANE];
    const T *qr = q + ((size_t)t * H + h) * d;
    float qv[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; i++) { const int c = lane + 32 * i; qv[i] = c < d ? to_f32(qr[c]) : 0.f; }

    const float slope = slopes ? slopes[h] : 0.f;
    if (head_scales) scale *= head_scales[h];
    const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;
    float m = -INFINITY, l = 0.f, acc[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; i++) acc[i] = 0.f;

    for (int j0 = lo + warp * KEYS; j0 <= pos; j0 += ATT_WARPS * KEYS) {
        // the cache rows of the group's keys, one a lane; -1: beyond the query, or no page
        long long row = -1;
        const int jl = j0 + lane;
        if (lane < KEYS && jl <= pos) {
            const int blk = jl / block_size;
            const long long page = blk < max_blocks ? table[blk] : -1;
            if (page < 0 || page >= num_pages) atomicOr(err, HFB_ERR_PAGE);
            else row = (page * block_size + (jl % block_size)) * G + g;
        }
        if (!__any_sync(0xffffffffu, row >= 0)) continue;            // (no page at all)
        float dot[KEYS], val[KEYS][PER_LANE];
#pragma unroll
        for (int i = 0; i < KEYS; i++) {
            const long long at = __shfl_sync(0xffffffffu, row, i);
            const T *kr = k_cache + at * d, *vr = v_cache + at * v_row;
            float x = 0.f;
#pragma unroll
            for (int e = 0; e < PER_LANE; e++) {
                const int c = lane + 32 * e;
                if (at >= 0 && c < d) x = fmaf(qv[e], to_f32(kr[c]), x);
                val[i][e] = at >= 0 && c < dv ? to_f32(vr[c]) : 0.f;
            }
            dot[i] = x;
        }
        float s = group_sum<KEYS>(dot) * scale;
        const int mine = key_of<KEYS>(lane);
        if (softcap > 0.f) s = softcap * tanhf(s * inv_cap);
        if (slopes) s -= slope * (float)(pos - (j0 + mine));
        if (__shfl_sync(0xffffffffu, row, mine) < 0) s = -INFINITY;
        float m_new = fmaxf(m, s);
#pragma unroll
        for (int o = 16; o >= 32 / KEYS; o >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
        const float corr = expf(m - m_new), p = expf(s - m_new);     // exp(-inf) = 0 on the first group
        float sum = p;
#pragma unroll
        for (int o = 16; o >= 32 / KEYS; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        l = l * corr + sum;
#pragma unroll
        for (int e = 0; e < PER_LANE; e++) acc[e] *= corr;
#pragma unroll
        for (int i = 0; i < KEYS; i++) {
            const float pi = __shfl_sync(0xffffffffu, p, lane_of<KEYS>(i));
#pragma unroll
            for (int e = 0; e < PER_LANE; e++) acc[e] = fmaf(pi, val[i][e], acc[e]);
        }
        m = m_new;
    }
    if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
#pragma unroll
    for (int i = 0; i < PER_LANE; i++) {
        int c = lane + 32 * i;
        if (c < dv) s_acc[warp][c] = acc[i];
    }
    __syncthreads();
    float mm = -INFINITY;
    for (int w = 0; w < ATT_WARPS; w++) mm = fmaxf(mm, s_m[w]);
    float ll = 0.f;
    float f[ATT_WARPS];
    for (int w = 0; w < ATT_WARPS; w++) {
        f[w] = s_m[w] == -INFINITY ? 0.f : expf(s_m[w] - mm);
        ll += s_l[w] * f[w];
    }
    float carry = 1.0f;                            // what the keys' share shrinks by when the sink is the largest score
    if (sinks || zero_sink) {
        const float sk = sinks ? sinks[h] : 0.f;
        const float top = fmaxf(mm, sk);
        carry = mm == -INFINITY ? 0.f : expf(mm - top);
        ll = ll * carry + expf(sk - top);
    }
    float inv = ll > 0.f ? carry / ll : 0.f;
    T *o = out + ((size_t)t * H + h) * dv;
    for (int c = threadIdx.x; c < dv; c += blockDim.x) {
        float v = 0.f;
        for (int w = 0; w < ATT_WARPS; w++) v += s_acc[w][c] * f[w];
        o[c] = from_f32<T>(v * inv);
    }
}

}  // namespace hfb

using namespace hfb;

extern "C" int hfb_attention_plain(const void *q, const void *k_cache, const void *v_cache, int dt,
                                   const int32_t *block_table, int max_blocks, const int32_t *token_seq,
                                   const int32_t *positions, int block_size, int64_t num_pages, int window,
                                   float scale, void *out, int T, int H, int G, int d, int dv, int v_row, const float *sinks,
                                   int zero_sink, const float *slopes, const float *head_scales, float softcap, hfb_stream s)
{
    if (T <= 0) return HFB_OK;
    if (!valid_dt(dt) || H <= 0 || G <= 0 || H % G || block_size <= 0 || max_blocks <= 0 || v_row < dv)
        return fail(HFB_EINVAL, "attention: bad arguments (H=%d G=%d block=%d)", H, G, block_size);
    if (d <= 0 || d > 32 * MAX_D_PER_LANE || dv <= 0 || dv > 32 * MAX_D_PER_LANE)
        return fail(HFB_ENOTSUP, "attention: head sizes %d / %d are not supported (1..%d)", d, dv, 32 * MAX_D_PER_LANE);
    if (H > 65535) return fail(HFB_ENOTSUP, "attention: %d heads exceed the grid limit", H);
    dim3 grid(T, H);
    const int wide = d > dv ? d : dv;
#define HFB_PLAIN_ATT(TY, L) \
    g_launch_err = launch_pdl(attention_plain_kernel<TY, L>, dim3(grid), dim3(ATT_WARPS * 32), 0, (cudaStream_t)s, (const TY *)q, (const TY *)k_cache, \
        (const TY *)v_cache, block_table, max_blocks, token_seq, positions, block_size, num_pages, window, scale, (TY *)out, H, G, d, dv, v_row, sinks, zero_sink, slopes, head_scales, softcap, error_word())
#define HFB_PLAIN_ATT_D(TY) \
    do { \
        if (wide <= 64) HFB_PLAIN_ATT(TY, 2); else if (wide <= 128) HFB_PLAIN_ATT(TY, 4); \
        else if (wide <= 256) HFB_PLAIN_ATT(TY, 8); else HFB_PLAIN_ATT(TY, MAX_D_PER_LANE); \
    } while (0)
    if (dt == HFB_F32) HFB_PLAIN_ATT_D(float);
    else HFB_PLAIN_ATT_D(__nv_bfloat16);
#undef HFB_PLAIN_ATT_D
#undef HFB_PLAIN_ATT
    return check_pdl_launch(g_launch_err, "attention_plain");
}
