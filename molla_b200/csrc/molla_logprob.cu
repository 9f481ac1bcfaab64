// Logprobs of the raw logits (sample.mojo:268-293) for rows of 4096 logits and more: the chosen token's,
// the top N's, or a whole row's. A tile of 1024 logits belongs to one warp, so a few rows fill the chip
// as well as many: one block per row, as for short rows, took 97 us for 64 rows of 151936 logits and left
// half of the SMs idle. 4096 is where a row has four tiles, fewer would leave most of a block of eight warps idle.
//
//   lp_tiles  every tile: its maximum and the sum of exp(z - maximum), accumulated in fp64
//                                           (bound: HBM, 4 bytes per logit, and an exponential per logit)
//   lp_rows   every row: maximum, logarithm of the sum, the chosen token, the top N. The N-th largest of
//             the tiles' maxima bounds the N-th largest logit from below, so only tiles whose maximum
//             reaches it, N of them but for ties, are looked at again
//   lp_whole  whole rows' logprobs, z - maximum - logarithm: a row per thread-block cluster
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include "molla_exact.cuh"
#include "molla_logprob.h"

namespace {

constexpr int LT_ = 256;          // threads of a block: eight warps, eight tiles
constexpr int LTILE = 1024;
constexpr int LREST = 64;         // a row's last piece of fewer logits goes with the tile before it
constexpr int LMAX_TILES = 704;
constexpr int LCAND = 512;

struct LpArgs {
    const float *logits; long long row_stride; int B, V;
    const int *tokens; int top_n; float *chosen; int *top_ids; float *top_lps;
    const int *rows; int n_logit_rows; float softcap;
    float *out;                   // whole rows' logprobs, or nullptr
    float *stats;                 // [rows][ntile] four floats
    bool early;                   // see lp_tiles
    int ntile;
};

__device__ __forceinline__ float *stat_of(const LpArgs &a, int r, int t) { return a.stats + ((long long)r * a.ntile + t) * 4; }
// which row of the block batch row r reads; -1 for a stale index (the row's sampling call has reported it)
__device__ __forceinline__ long long logit_row(const LpArgs &a, int r) {
    const long long l = a.rows ? (long long)a.rows[r] : (long long)r;
    return (a.rows && (l < 0 || (a.n_logit_rows > 0 && l >= a.n_logit_rows))) ? -1 : l;
}
__device__ __forceinline__ int tile_end(const LpArgs &a, int t) { return t == a.ntile - 1 ? a.V : (t + 1) * LTILE; }
// A tile of n logits (the row's last one up to 64 more than LTILE) by one warp: by sixteen bytes a lane where `wide`
// and the tile is whole, by words elsewhere; `none` for what is not there. Returns which.
__device__ __forceinline__ bool load_tile(float (&x)[34], const float *z, int n, int lane, bool wide, float none) {
    wide = wide && n >= LTILE;
    if (wide) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(z) + lane + 32 * i);
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; i++) x[i] = lane + 32 * i < n ? __ldg(z + lane + 32 * i) : none;
    }
    x[32] = LTILE + lane < n ? __ldg(z + LTILE + lane) : none;
    x[33] = LTILE + 32 + lane < n ? __ldg(z + LTILE + 32 + lane) : none;
    return wide;
}
__device__ __forceinline__ float capped(const LpArgs &a, float x) { return a.softcap > 0.0f ? softcap_pinned(x, a.softcap) : x; }

// A tile's maximum and its sum of exp(z - maximum) in fp64, one warp.
__device__ __forceinline__ void tile_stat(const float (&x)[34], float &m, double &sum) {
    m = -INFINITY;
#pragma unroll
    for (int i = 0; i < 34; i++) m = fmaxf(m, x[i]);
    m = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(m)));
    double s0 = 0.0, s1 = 0.0;
    if (m > -INFINITY) {
#pragma unroll
        for (int i = 0; i < 34; i += 2) {
            s0 += (double)expf_pinned_nonpos(__fsub_rn(x[i], m));
            s1 += (double)expf_pinned_nonpos(__fsub_rn(x[i + 1], m));
        }
    }
    s0 += s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    sum = s0;
}

__device__ __forceinline__ void lp_tile(const LpArgs &a) {
    const int lane = threadIdx.x & 31, per = (a.ntile + 7) / 8;
    const int r = blockIdx.x / per, t = (blockIdx.x - r * per) * 8 + (threadIdx.x >> 5);
    if (t >= a.ntile) return;
    const long long lrow = logit_row(a, r);
    if (lrow < 0) return;
    const float *z = a.logits + lrow * a.row_stride + (long long)t * LTILE;
    const int n = tile_end(a, t) - t * LTILE;
    float x[34];
    (void)load_tile(x, z, n, lane, (reinterpret_cast<uintptr_t>(z) & 15u) == 0, -INFINITY);
    if (a.softcap > 0.0f) {
#pragma unroll
        for (int i = 0; i < 34; i++) if (x[i] > -INFINITY) x[i] = softcap_pinned(x[i], a.softcap);
    }
    float m;
    double s0;
    tile_stat(x, m, s0);
    if (lane == 0) {
        float *o = stat_of(a, r, t);
        const unsigned long long b = (unsigned long long)__double_as_longlong(s0);
        o[0] = m; o[1] = __uint_as_float((unsigned int)b); o[2] = __uint_as_float((unsigned int)(b >> 32));
    }
}

// `early`: this kernel may run beside the one before it, which nothing here depends on (the logits are older, and it does
// not touch a.stats). The kernel behind this one needs that one's tokens: so it ends only when that one has, which
// one block waits for.
__global__ void __launch_bounds__(LT_) lp_tiles(const __grid_constant__ LpArgs a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!a.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    lp_tile(a);
    if (a.early && blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

__global__ void __launch_bounds__(LT_) lp_rows(const __grid_constant__ LpArgs a) {
    __shared__ float tm[LMAX_TILES];
    __shared__ unsigned short pick[LMAX_TILES];
    __shared__ unsigned long long cand[LCAND];
    __shared__ double wsd[LT_ / 32];
    __shared__ float wsf[LT_ / 32];
    __shared__ int wsi[LT_ / 32];
    __shared__ int npick, ncand;
    __shared__ float s_thr;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, top_n = a.top_n;
    const long long lrow = logit_row(a, r);
    if (lrow < 0) {
        if (a.chosen && tid == 0) a.chosen[r] = 0.0f;
        for (int i = tid; i < top_n; i += LT_) { a.top_ids[(long long)r * top_n + i] = -1; a.top_lps[(long long)r * top_n + i] = 0.0f; }
        return;
    }
    const float *z = a.logits + lrow * a.row_stride;
    constexpr int PER = (LMAX_TILES + LT_ - 1) / LT_;
    double sum[PER];
    float m[PER], top = -INFINITY;
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int t = tid + u * LT_;
        sum[u] = 0.0; m[u] = -INFINITY;
        if (t < a.ntile) {
            const float *o = stat_of(a, r, t);
            m[u] = o[0];
            sum[u] = __longlong_as_double((long long)((unsigned long long)__float_as_uint(o[1]) | ((unsigned long long)__float_as_uint(o[2]) << 32)));
            tm[t] = m[u];
        }
        top = fmaxf(top, m[u]);
    }
    top = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(top)));
    if (lane == 0) wsf[warp] = top;
    if (tid == 0) { npick = 0; ncand = 0; s_thr = -INFINITY; }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < LT_ / 32; w++) top = fmaxf(top, wsf[w]);
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < PER; u++)
        if (m[u] > -INFINITY) s += sum[u] * exp((double)m[u] - (double)top);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) wsd[warp] = s;
    __syncthreads();
    s = 0.0;
#pragma unroll
    for (int w = 0; w < LT_ / 32; w++) s += wsd[w];
    const float offset = (float)log(s);
    if (a.chosen && a.tokens && tid == 0) {
        const int t = a.tokens[r];
        a.chosen[r] = (t >= 0 && t < a.V) ? __fsub_rn(__fsub_rn(capped(a, __ldg(z + t)), top), offset) : 0.0f;
    }
    if (top_n == 0) return;
    // the tiles whose maximum is among the top_n largest; equal maxima count in order
    if (a.ntile >= top_n) {
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int t = tid + u * LT_;
            if (t >= a.ntile) break;
            int above = 0;
            for (int o = 0; o < a.ntile; o++) above += (tm[o] > m[u] || (tm[o] == m[u] && o < t)) ? 1 : 0;
            if (above == top_n - 1) s_thr = m[u];
        }
    }
    __syncthreads();
    const float thr = s_thr;
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int t = tid + u * LT_;
        if (t < a.ntile && m[u] >= thr) pick[satom_add(&npick, 1)] = (unsigned short)t;
    }
    __syncthreads();
    for (int i = warp; i < npick; i += LT_ / 32) {
        const int t = pick[i], e1 = tile_end(a, t);
        for (int e = t * LTILE + lane; e < e1; e += 32 * 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = e + 32 * u < e1 ? __ldg(z + e + 32 * u) : -INFINITY;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (e + 32 * u >= e1) continue;
                const float x = capped(a, v[u]);
                if (x >= thr) {
                    const int pos = satom_add(&ncand, 1);
                    if (pos < LCAND) cand[pos] = ((unsigned long long)fkey(x) << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned int)(e + 32 * u));
                }
            }
        }
    }
    __syncthreads();
    const int n = ncand;
    if (n <= LCAND) {
        for (int i = tid; i < n; i += LT_) {
            const unsigned long long mine = cand[i];
            int rank = 0;
            for (int j = 0; j < n; j++) rank += cand[j] > mine ? 1 : 0;
            if (rank < top_n) {
                const int id = (int)(0xFFFFFFFFu - (unsigned int)(mine & 0xFFFFFFFFull));
                a.top_ids[(long long)r * top_n + rank] = id;
                a.top_lps[(long long)r * top_n + rank] = __fsub_rn(__fsub_rn(fkey_inv((unsigned int)(mine >> 32)), top), offset);
            }
        }
        for (int i = n + tid; i < top_n; i += LT_) { a.top_ids[(long long)r * top_n + i] = -1; a.top_lps[(long long)r * top_n + i] = 0.0f; }
        return;
    }
    // More logits at or above the threshold than the buffer holds (a flat or heavily quantised row): the N
    // largest one after the other, each the first in the order (value descending, index ascending) behind
    // the one before it. A pass per pick.
    float lastv = INFINITY;
    int lasti = -1;
    for (int k = 0; k < top_n; k++) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int i = tid; i < a.V; i += LT_) {
            const float x = capped(a, __ldg(z + i));
            const bool behind = x < lastv || (x == lastv && i > lasti);
            if (behind && (x > bv || (x == bv && i < bi))) { bv = x; bi = i; }
        }
        warp_argmax(bv, bi);
        __syncthreads();
        if (lane == 0) { wsf[warp] = bv; wsi[warp] = bi; }
        __syncthreads();
        bv = wsf[0]; bi = wsi[0];
        for (int w = 1; w < LT_ / 32; w++)
            if (wsf[w] > bv || (wsf[w] == bv && wsi[w] < bi)) { bv = wsf[w]; bi = wsi[w]; }
        const bool found = bi != 0x7fffffff;
        if (tid == 0) {
            a.top_ids[(long long)r * top_n + k] = found ? bi : -1;
            a.top_lps[(long long)r * top_n + k] = found ? __fsub_rn(__fsub_rn(bv, top), offset) : 0.0f;
        }
        lastv = bv; lasti = bi;
        if (!found) lastv = -INFINITY;
    }
}

// A whole row's logprobs, one cluster: every block its tiles' maxima and sums, those of all blocks through distributed
// shared memory, then the same tiles again, which are in L2 (the clusters in flight hold some 300 bytes per logit of
// the vocabulary), and the result. Bound: the exponentials' instructions, then the store. One launch: with a kernel
// for the tiles, one for the rows and one for the result, 64 rows of 128256 took 22.0 us, now 19.5 (floor 10), 512 of
// 262144 285 and 221, 16 of 32000 12.5 and 8.1. Clusters of sixteen where rows are few or
// widest (molla_logprob_launch): 7 rows of 700000 took 21.8 us in clusters of eight, 13.8 of sixteen.
constexpr int LG_MOST = 16;
__global__ void __launch_bounds__(512, 2) lp_whole(const __grid_constant__ LpArgs a) {
    namespace cg = cooperative_groups;
    __shared__ float tm[LMAX_TILES], bm[LG_MOST], s_top, s_off;
    __shared__ double ts[LMAX_TILES], bs[LG_MOST];
    cg::cluster_group cl = cg::this_cluster();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    cluster_begun();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (int)blockDim.x >> 5, G = (int)cl.num_blocks(), rank = (int)cl.block_rank(), r = (int)blockIdx.x / G;
    const int per = (a.ntile + G - 1) / G, t0 = rank * per, n = max(0, min(per, a.ntile - t0));
    const float *z = a.logits + (long long)r * a.row_stride + (long long)t0 * LTILE;
    float *o = a.out + (long long)r * a.V + (long long)t0 * LTILE;
    const bool in16 = (reinterpret_cast<uintptr_t>(z) & 15u) == 0, out16 = (reinterpret_cast<uintptr_t>(o) & 15u) == 0;
    float x[34];
#pragma unroll 1
    for (int t = warp; t < n; t += warps) {
        (void)load_tile(x, z + t * LTILE, tile_end(a, t0 + t) - (t0 + t) * LTILE, lane, in16, -INFINITY);
        float m;
        double s;
        tile_stat(x, m, s);
        if (lane == 0) { tm[t] = m; ts[t] = s; }
    }
    __syncwarp();
    cluster_all_begun();   // (blocks without tiles get here at once)
    __syncthreads();
    if (warp == 0) {
        float m = -INFINITY;
        for (int t = lane; t < n; t += 32) m = fmaxf(m, tm[t]);
        m = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(m)));
        double s = 0.0;
        for (int t = lane; t < n; t += 32)
            if (tm[t] > -INFINITY) s += ts[t] * exp((double)tm[t] - (double)m);
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) s += __shfl_xor_sync(0xffffffffu, s, i);
        if (lane < G) { *cl.map_shared_rank(&bm[rank], lane) = m; *cl.map_shared_rank(&bs[rank], lane) = s; }
    }
    cl.sync();
    if (warp == 0) {
        const float m = lane < G ? bm[lane] : -INFINITY, top = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(m)));
        double s = m > -INFINITY ? bs[lane] * exp((double)m - (double)top) : 0.0;
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) s += __shfl_xor_sync(0xffffffffu, s, i);
        if (lane == 0) { s_top = top; s_off = (float)log(s); }
    }
    __syncthreads();
    const float top = s_top, offset = s_off;
#pragma unroll 1
    for (int t = warp; t < n; t += warps) {
        const int e = tile_end(a, t0 + t) - (t0 + t) * LTILE;
        float *to = o + t * LTILE;
        const bool vec = load_tile(x, z + t * LTILE, e, lane, in16 && out16, 0.0f);
#pragma unroll
        for (int i = 0; i < 34; i++) x[i] = __fsub_rn(__fsub_rn(x[i], top), offset);
        if (vec) {
#pragma unroll
            for (int i = 0; i < 8; i++) __stcs(reinterpret_cast<float4 *>(to) + lane + 32 * i, make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]));
        } else {
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (lane + 32 * i < e) __stcs(to + lane + 32 * i, x[i]);
        }
        if (LTILE + lane < e) to[LTILE + lane] = x[32];
        if (LTILE + 32 + lane < e) to[LTILE + 32 + lane] = x[33];
    }
}

void lp_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, unsigned int blocks, unsigned int threads, unsigned int cluster, cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(blocks); cfg.blockDim = dim3(threads); cfg.stream = st;
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = cluster > 1 ? 2 : 1;
}
cudaError_t lp_launch(void (*kernel)(LpArgs), unsigned int blocks, unsigned int threads, unsigned int cluster, cudaStream_t st, const LpArgs &a) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    lp_config(cfg, at, blocks, threads, cluster, st);
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

// Whether this device takes lp_whole's clusters of sixteen, which no device has to (asked once per device).
bool wide_clusters(int dev) {
    constexpr int DEVICES = 64;
    static int known[DEVICES] = {};  // 0 unknown, -1 no
    if (dev < 0 || dev >= DEVICES) return false;
    if (known[dev] == 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        lp_config(cfg, at, LG_MOST, 512, LG_MOST, nullptr);
        int n = 0;
        const bool ok = cudaFuncSetAttribute(lp_whole, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, lp_whole, &cfg) == cudaSuccess && n > 0;
        if (!ok) (void)cudaGetLastError();
        known[dev] = ok ? 1 : -1;
    }
    return known[dev] > 0;
}

int tiles_of(int V) {
    const int full = V / LTILE, rest = V % LTILE;
    return full + (rest >= LREST ? 1 : 0);
}

}  // namespace

// (with fewer tiles than the top N asks for, no tile's maximum bounds the N-th largest: the scan that is
// then left took 38 us for 13 rows of 5248 and a top 20, the one block a row of short rows 20)
bool molla_logprob_tiled(int V, int top_n) { return V >= 4096 && tiles_of(V) >= top_n && tiles_of(V) <= LMAX_TILES; }
size_t molla_logprob_workspace_bytes(int B, int V) { return (size_t)B * (size_t)tiles_of(V) * 4 * sizeof(float); }

cudaError_t molla_logprob_launch(const float *logits, long long row_stride, int B, int V, const int *tokens, int top_n, float *chosen,
                                 int *top_ids, float *top_lps, const int *rows, int n_logit_rows, float softcap, void *workspace, bool early,
                                 float *full_out, bool wide, cudaStream_t st) {
    LpArgs a = {};
    a.logits = logits; a.row_stride = row_stride; a.B = B; a.V = V;
    a.tokens = tokens; a.top_n = top_n; a.chosen = chosen; a.top_ids = top_ids; a.top_lps = top_lps;
    a.rows = rows; a.n_logit_rows = n_logit_rows; a.softcap = softcap; a.out = full_out;
    a.ntile = tiles_of(V);
    if (full_out) {
        // A block for eight tiles, up to eight of them; sixteen for the widest rows and for few; as many warps as
        // share a block's tiles evenly in rounds of at most eight, of sixteen where there are not two blocks an SM.
        // Few rows: those whose blocks, at eight a row, are three an SM at most on the SMs that clusters of eight reach (8/9 of
        // them). (At two an SM, 48 rows of 140000 had clusters of eight, 18 tiles a block in three rounds of six: 24.0 us, where
        // sixteen of nine tiles in two rounds take 18.3; 38 of 128256 18.2 and 14.7, 40 of 196000 25.4 and 19.8.) Where they are
        // four an SM a block has seven warps at least, so that no SM takes a fifth: 64 of 140000 24.4 and 22.0, of 90000 17.4 and 15.2.
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) { dev = -1; sms = 0; }
        int G = 1;
        while (G < 8 && 8 * G < a.ntile) G *= 2;
        const long long reached = (long long)sms * 8 / 9;
        if ((a.ntile > 24 * 8 || (a.ntile > 8 * 8 && (long long)B * G <= 3 * reached)) && wide && wide_clusters(dev)) G = LG_MOST;
        const long long n = (long long)B * G;
        const int each = (a.ntile + G - 1) / G, most = n <= 2 * sms ? 16 : 8, rounds = (each + most - 1) / most;
        int warps = (each + rounds - 1) / rounds;
        if (n > 3 * reached && n <= 4 * reached && warps < 7) warps = each < 7 ? each : 7;
        return lp_launch(lp_whole, (unsigned int)n, 32u * (unsigned int)warps, (unsigned int)G, st, a);
    }
    a.stats = (float *)workspace; a.early = early;
    const unsigned int blocks = (unsigned int)B * (unsigned int)((a.ntile + 7) / 8);
    cudaError_t e = lp_launch(lp_tiles, blocks, LT_, 1, st, a);
    if (e == cudaSuccess) e = lp_launch(lp_rows, (unsigned int)B, LT_, 1, st, a);
    return e;
}
