// The grouped product of a mixture of experts for tiles of many places, on the 5th-generation tensor cores:
// out[dst(p), :] = act(a[src(p), :] . w[expert(p)]^T), bfloat16 operands, float32 accumulators.
//
// A work item is 128 features of one expert (accumulator rows) by the up to 256 places of one tile of the lists
// (accumulator columns).  The number of columns is the tile's own, rounded up to 16: experts get as many tokens as the
// router sends them, and a fixed tile of tokens would multiply padding (an expert with 140 places costs 144 columns here,
// two tiles of 128 before).  The weights stream through the rows once per tile.  The places' rows lie one behind the other
// and come in boxes of 32: the down product's do anyway, the up product's are copied so by a small kernel first (TMA
// gathers of four rows each took 60 ns an instruction: 1,109 us for 9,000 places of 4,096 x 3,072).  Rows that a box
// brings from behind the tile are multiplied at most and not stored.
// Persistent blocks walk the items, features first, so that a tile's places come from L2 after the first item; one warp
// requests weights, one the places, one issues tcgen05.mma into one of two accumulators, eight drain the other.
// What bounds it: at 280 places an expert the tensor cores, at a few tens the weight stream.
// Measured (B200, 32 experts; mma.sync tiles of 128 x 128 before): 8,192 places, up 1,024 x 2,048 with the copy 208 -> 64
// us, down 204 -> 57 us (607 TFLOP/s); 9,000 places, gated up 3,072 x 4,096 1,059 -> 303 us (748 TFLOP/s), down 587 -> 148
// us; 800 places (25 an expert) 80 -> 33 us, which streams the weights at 4.1 TB/s.
#include <cuda.h>

#include "moe_common.cuh"
#include "tc_ptx.cuh"

static thread_local cudaError_t g_launch_err = cudaSuccess;      // what the last launch_pdl returned

namespace hfb {
int *error_word();
int tensor_map(const void *ptr, int rows, int cols, int box_rows, CUtensorMap *out);

constexpr int MG_K = 64, MG_X = 128, MG_Y = 256, MG_STAGES = 4, MG_BOX = 32;
constexpr uint32_t MG_XB = MG_X * MG_K * 2, MG_YB = MG_Y * MG_K * 2;
constexpr uint32_t MG_SMEM = 1024 + MG_STAGES * (MG_XB + MG_YB) + (2 * MG_STAGES + 4) * 8 + 16;
constexpr int MG_THREADS = 352;              // weight warp, MMA warp, eight epilogue warps, places warp
constexpr int MG_PLACES_WARP = 10;

struct MoeTcParams {
    int N, K, f_tiles;                       // features of an expert, inner size, tiles of 128 features
    int scatter, act, glu;
    GluClamp clamp;
    void *out; int out_dt;
    const int32_t *order, *tile_expert, *tile_p0, *tile_n, *n_tiles;
};

// The activations of 32 values at once: the choice is made outside the loops (inside them the code of all activations,
// 32 times over, does not fit the instruction cache, and every value waits for its next lines behind the weight stream).
__device__ __forceinline__ void moe_tc_act(float (&z)[32], int act)
{
    if (act == HFB_ACT_RELU2) {
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = moe_act(z[i], HFB_ACT_RELU2);
    } else if (act == HFB_ACT_RELU) {
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = moe_act(z[i], HFB_ACT_RELU);
    } else if (act == HFB_ACT_SILU) {
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = moe_act(z[i], HFB_ACT_SILU);
    } else if (act == HFB_ACT_GELU_TANH) {
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = moe_act(z[i], HFB_ACT_GELU_TANH);
    }
}

// 32 columns (places c0 ..) of one accumulator row (feature f); `live` places exist, lane l knows the row of the output of
// place c0 + l.
__device__ __forceinline__ void moe_tc_store(const MoeTcParams &p, float (&z)[32], int f, int live, int dst_l, int lane)
{
    const bool bf = p.out_dt == HFB_BF16;
    if (p.glu) {
        // rows alternate gate, up: the two lanes of a pair exchange values, the even one finishes the first of every two
        // places, the odd one the second
        const int odd = lane & 1, ldo = p.N >> 1;
        float h[16];
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const float other = __shfl_xor_sync(0xffffffffu, odd ? z[2 * j] : z[2 * j + 1], 1);
            const float mine = odd ? z[2 * j + 1] : z[2 * j];
            z[2 * j] = odd ? other : mine;                   // gate
            z[2 * j + 1] = odd ? mine : other;               // up
        }
        if (p.act == HFB_ACT_CLAMPED_GLU) {
#pragma unroll
            for (int j = 0; j < 16; j++) h[j] = moe_glu(z[2 * j], z[2 * j + 1], HFB_ACT_CLAMPED_GLU, p.clamp);
        } else if (p.act == HFB_ACT_SILU) {
#pragma unroll
            for (int j = 0; j < 16; j++) h[j] = moe_glu(z[2 * j], z[2 * j + 1], HFB_ACT_SILU, p.clamp);
        } else {
#pragma unroll
            for (int j = 0; j < 16; j++) h[j] = moe_glu(z[2 * j], z[2 * j + 1], p.act, p.clamp);
        }
        const bool in = (f | 1) < p.N;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            if (2 * j >= live) break;                        // (the same for the whole warp)
            const int i = 2 * j + odd, dst = __shfl_sync(0xffffffffu, dst_l, i);
            if (in && i < live) {
                const size_t at = (size_t)dst * ldo + (f >> 1);
                if (bf) ((__nv_bfloat16 *)p.out)[at] = __float2bfloat16_rn(h[j]);
                else ((float *)p.out)[at] = h[j];
            }
        }
        return;
    }
    moe_tc_act(z, p.act);
    const bool in = f < p.N;
    if (bf) {
        __nv_bfloat16 *out = (__nv_bfloat16 *)p.out + f;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            if (i >= live) break;
            const int dst = __shfl_sync(0xffffffffu, dst_l, i);
            if (in) out[(size_t)dst * p.N] = __float2bfloat16_rn(z[i]);
        }
    } else {
        float *out = (float *)p.out + f;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            if (i >= live) break;
            const int dst = __shfl_sync(0xffffffffu, dst_l, i);
            if (in) out[(size_t)dst * p.N] = z[i];
        }
    }
}

// rows[p, :] = a[order[p] / src_div, :]: the places' rows one behind the other, sixteen bytes a thread.  (Entries of order
// behind the last place are whatever they are: they are kept in range, and nothing reads their rows.)
__global__ void moe_gather_kernel(const uint4 *a, const int32_t *order, int src_div, uint4 *rows, int pairs, int pieces)
{
    pdl_sync();
    const size_t total = (size_t)pairs * pieces;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int p = (int)(i / pieces), c = (int)(i % pieces);
        const int pair = order[p];
        if ((unsigned)pair < (unsigned)pairs) rows[i] = a[(size_t)(pair / src_div) * pieces + c];
    }
}

__global__ void __launch_bounds__(MG_THREADS, 1)
moe_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, MoeTcParams p, int *err)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t sx = base, sy = base + MG_STAGES * MG_XB, bars = sy + MG_STAGES * MG_YB;
    const uint32_t full0 = bars, empty0 = bars + MG_STAGES * 8, tfull0 = bars + 2 * MG_STAGES * 8, tempty0 = tfull0 + 16;
    uint8_t *gen_base = smem_raw + (base - smem_u32(smem_raw));
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(gen_base + MG_STAGES * (MG_XB + MG_YB) + (2 * MG_STAGES + 4) * 8);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < MG_STAGES; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int a = 0; a < 2; a++) { mbar_init(tfull0 + 8 * a, 1); mbar_init(tempty0 + 8 * a, 8); }       // eight epilogue warps
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32((const void *)tmem_slot)), "r"(2 * MG_Y) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    pdl_sync();                                              // the lists themselves come from the kernels in front
    const int items = *p.n_tiles * p.f_tiles, kbs = (p.K + MG_K - 1) / MG_K;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
                const int ti = item / p.f_tiles, ft = item % p.f_tiles;
                const int row = p.tile_expert[ti] * p.N + ft * MG_X;
                const uint32_t bytes = MG_XB + (uint32_t)((p.tile_n[ti] + MG_BOX - 1) / MG_BOX) * (MG_BOX * MG_K * 2);
                for (int kb = 0; kb < kbs; kb++, it++) {
                    const int s = it % MG_STAGES;
                    if (!mbar_wait(empty0 + 8 * s, ((it / MG_STAGES) & 1) ^ 1, abort_flag, err)) { ok = false; break; }
                    mbar_arrive_expect_tx(full0 + 8 * s, bytes);
                    tma_load_2d(sx + s * MG_XB, &map_w, kb * MG_K, row, full0 + 8 * s);
                }
            }
        }
    } else if (warp == MG_PLACES_WARP) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
                const int ti = item / p.f_tiles, p0 = p.tile_p0[ti], rows = p.tile_n[ti];
                for (int kb = 0; kb < kbs; kb++, it++) {
                    const int s = it % MG_STAGES;
                    if (!mbar_wait(empty0 + 8 * s, ((it / MG_STAGES) & 1) ^ 1, abort_flag, err)) { ok = false; break; }
                    for (int r = 0; r < rows; r += MG_BOX)
                        tma_load_2d(sy + s * MG_YB + r * (MG_K * 2), &map_a, kb * MG_K, p0 + r, full0 + 8 * s);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t it = 0, tile_it = 0, last_ph = 0;
            int last_s = -1;
            bool ok = true;
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x, tile_it++) {
                const uint32_t idesc = bf16_idesc(MG_X, (p.tile_n[item / p.f_tiles] + 15) & ~15, false);
                const int a = tile_it & 1;
                if (!mbar_wait(tempty0 + 8 * a, ((tile_it >> 1) & 1) ^ 1, abort_flag, err)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem_base + a * MG_Y;
                for (int kb = 0; kb < kbs; kb++, it++) {
                    const int s = it % MG_STAGES;
                    const uint32_t ph = (it / MG_STAGES) & 1;
                    if (!mbar_wait(full0 + 8 * s, ph, abort_flag, err)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t dx = sw128_desc(sx + s * MG_XB), dy = sw128_desc(sy + s * MG_YB);
#pragma unroll
                    for (int k = 0; k < MG_K / 16; k++) tc_mma_bf16(d, dx + 2 * k, dy + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit(empty0 + 8 * s);
                    last_s = s;
                    last_ph = ph;
                }
                if (ok) tc_commit(tfull0 + 8 * a);
            }
            if (ok && last_s >= 0) mbar_wait(empty0 + 8 * last_s, last_ph, abort_flag, err);
        }
    } else {
        // two warps for each quarter of the accumulator's lanes, every second 32 of its columns each
        const int q = warp & 3, row = q * 32 + lane;
        uint32_t tile_it = 0;
        for (int item = blockIdx.x; item < items; item += gridDim.x, tile_it++) {
            const int ti = item / p.f_tiles, f = (item % p.f_tiles) * MG_X + row;
            const int p0 = p.tile_p0[ti], rows = p.tile_n[ti], a = tile_it & 1;
            if (!mbar_wait_long(tfull0 + 8 * a, (tile_it >> 1) & 1, abort_flag, err)) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + a * MG_Y;
#pragma unroll 1
            for (int c0 = warp >= 6 ? 32 : 0; c0 < rows; c0 += 64) {
                uint32_t v[32];
                tmem_ld16(taddr + c0, v);
                tmem_ld16(taddr + c0 + 16, v + 16);
                const int place = p0 + min(c0 + lane, rows - 1);
                const int dst = p.scatter ? p.order[place] : place;
                tmem_wait_ld();
                float z[32];
#pragma unroll
                for (int i = 0; i < 32; i++) z[i] = __uint_as_float(v[i]);
                moe_tc_store(p, z, f, min(32, rows - c0), dst, lane);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty0 + 8 * a);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // a wait ran out: give loads that are still in flight time to land before the shared memory goes away
        for (int i = 0; i < 2000; i++) __nanosleep(1000);
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * MG_Y) : "memory");
    }
}

// Called by hfb_moe_gemm, which has checked the arguments: K a multiple of 8, operands 16-byte aligned, tiles of up to 256
// places.  `a` holds the places' rows one behind the other (a_rows of them), or with src_div > 0 the tokens' rows, which are
// then laid out so in `rows` ([a_rows * src_div, K]) first; `experts`: matrices in w.
int moe_gemm_tc(const void *a, int a_rows, void *rows, const void *w, int experts, void *out, int out_dt, int act, const GluClamp &clamp, int N, int K,
                const int32_t *order, int src_div, int scatter, const int32_t *tile_expert, const int32_t *tile_p0,
                const int32_t *tile_n, const int32_t *n_tiles, int max_tiles, cudaStream_t st)
{
    static bool opted[64] = {};                  // more than 48 KB of shared memory: asked for once per device
    static int sms[64] = {};
    const int dev = current_device();
    if (!opted[dev]) {
        if (cudaFuncSetAttribute(moe_gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MG_SMEM) != cudaSuccess)
            return fail(HFB_ECUDA, "moe_gemm: the kernel's shared memory could not be set");
        cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        opted[dev] = true;
    }
    if (src_div > 0) {
        const int pairs = a_rows * src_div, pieces = K / 8;
        const size_t blocks = ((size_t)pairs * pieces + 255) / 256;
        g_launch_err = launch_pdl(moe_gather_kernel, dim3((unsigned)(blocks < 148 * 16 ? blocks : 148 * 16)), dim3(256), 0, st, (const uint4 *)a, order, src_div,
                                  (uint4 *)rows, pairs, pieces);
        const int rc = check_pdl_launch(g_launch_err, "moe_gather");
        if (rc != HFB_OK) return rc;
        a = rows;
        a_rows = pairs;
    }
    CUtensorMap mw, ma;
    int rc = tensor_map(w, experts * N, K, MG_X, &mw);
    if (rc == HFB_OK) rc = tensor_map(a, a_rows, K, MG_BOX, &ma);
    if (rc != HFB_OK) return rc;
    MoeTcParams p{};
    p.N = N; p.K = K; p.f_tiles = (N + MG_X - 1) / MG_X;
    p.scatter = scatter; p.act = act & 255; p.glu = act >> 8; p.clamp = clamp;
    p.out = out; p.out_dt = out_dt;
    p.order = order; p.tile_expert = tile_expert; p.tile_p0 = tile_p0; p.tile_n = tile_n; p.n_tiles = n_tiles;
    const long long most = (long long)max_tiles * p.f_tiles;
    const int grid = (int)(most < sms[dev] ? most : sms[dev] > 0 ? sms[dev] : 1);
    g_launch_err = launch_pdl(moe_gemm_tc_kernel, dim3(grid), dim3(MG_THREADS), MG_SMEM, st, mw, ma, p, error_word());
    return check_pdl_launch(g_launch_err, "moe_gemm_tc");
}

}  // namespace hfb
