// The ordinary entry points' path for batches whose rows do not all fit the chip at once in thread-block
// clusters: seven small kernels.
//
//   tile_stats   every tile of 1024 logits: its maximum, where it lies, and an estimate of the tile's
//                sum of exponentials                                     (reads the block from HBM)
//   row_plan     every row: the maximum, the answer of greedy rows, an estimate of the running softmax
//                sum before every tile, what is too small to matter there, and a value that the
//                `need` largest elements reach
//   tile_exp     every tile again (from L2 where the block fits it): the exponentials of what can
//                matter, the head's candidates, and a short program ("items") that says how the exact
//                sequential sum goes through the tile
//   row_head     every row: one warp runs the items, which gives the exact softmax denominator, then
//                the sorted head, the filters and the draw; most rows end here, the others are queued
//   tile_walk    queued rows, every tile: probabilities, and either the items of their sum (nothing is
//                sorted) or the bin tables of the walk past the head; the last block of a row chooses
//                the bins that the walk will look into
//   tile_pick    queued rows, every tile: the elements of those bins
//   row_tail     queued rows: the rest of the walk and of the draw, and the general form of everything
//
// A tile belongs to one warp and no warp waits for another (except around bias and penalty patches),
// so any number of rows, from one to thousands, fills the chip, and only the row kernels have serial
// parts. A row per thread-block cluster, resident in its shared memory, read the block once but left 33 to 16
// rows in flight on the chip, each as slow as its serial parts: 1024 rows of 262144 took 6316 us where this
// takes 690 to 700, 64 of 151936 with a nucleus and logprobs 300 where this takes 168 to 184. Seven launches cost 2 to 3 us each where
// nothing else is to be done; they are chained so that a kernel's blocks are in place when the one before
// ends. The reference's sequential fp32 sums are reproduced bit for bit: see "Items" below.
#include <cuda_runtime.h>
#include <math.h>
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>

#include "molla_exact.cuh"
#include "molla_rows.h"

namespace {

constexpr int TILE = 1024;                 // logits of a tile: 32 per lane, consecutive
constexpr int PITCH = 36;                  // words per lane in shared memory: float4 accesses without bank conflicts
constexpr int SPAN_THREADS = 256;          // a block of the tile kernels: eight warps, eight tiles
constexpr int SPAN = SPAN_THREADS * 32;    // logits per block
constexpr int MAX_TILES = 704;             // V <= 720896
constexpr int ITEMS_PER_TILE = 66;         // a run and a careful chunk per lane at most, and one more run
constexpr int ITEM_CAP = 384;              // items of a row that fit shared memory
constexpr int CARE_PLACES = 255;           // careful chunks of a row whose values are handed on with the items
constexpr int CARE_CAP = 48;               // careful chunks whose entries are fetched ahead
constexpr int TIE_CAP = 64;                // rounding ties a walk resolves by parity; more send it the slow way
constexpr int PLAN_BINS = 1024;            // row_plan: bins of the lanes' maxima by distance below the row's,
constexpr float PLAN_RES = 32.0f;          // 32 per unit of logit

enum { PLAN_DONE = 0, PLAN_SAMPLED = 1 };
enum { F_LIST = 1, F_FASTDIV = 2, F_PURE = 4, F_NARROW = 8, F_JUMP = 16, F_FAR = 32, F_ALLNEAR = 64 };

// The far head. A row without a top-k sorts what at least HEAD_NEED lanes' maxima reach and walks on through
// tables of its list where top-p lies behind that: three more kernels, 60 to 80 us however short the row. In
// rows of up to FAR_MOST_V logits most nuclei end within about FAR_HEAD elements, so their candidates go further
// down: those the head has had all along (near) in one list, the others in a second one, used where both fit the
// head's buffer together. Longer rows keep the near head: at 151936 seven nuclei in ten end behind either.
// F_ALLNEAR: the row has fewer lanes than its head wants elements, or hardly more, so the near list mostly holds too
// much; the second one, which ends higher up, is then the head alone, if it holds what a top-k asks for (aimed at
// FAR_TOPK elements, between that and the buffer's size).
// Without and with it, us: 512 rows with mixed settings, 4000 logits 156 / 139, 8000 158 / 142, 20000 193 / 175;
// 256 rows with a nucleus, 4000 logits 169 / 64, 8000 150 / 69, 20000 192 / 131, 50257 266 / 200;
// with a top-k of 1024, 8000 169 / 128, 20000 290 / 100.
constexpr int FAR_MOST_V = 65536, FAR_HEAD = 1000, FAR_TOPK = 1450;

struct __align__(16) TileStat { float tmax, tsum; int tidx, teq; };
struct __align__(8) TilePlan { float thr, est; };
struct __align__(8) TileOut { unsigned int ioff; unsigned short cnt, nitem; };   // its items in the row's, entries in its list

// Items: the exact sequential sum of a tile's values as a short program. While the running sum s
// stays in one binade, fl(s + v) is s plus rne(v / ulp) units; in the bit pattern of s, adding k units is
// the integer addition of k. Only where v / ulp ends in a half (a rounding tie) does the integer depend on s,
// and then only on the parity of its bit pattern. So any stretch of values is two numbers, the units it adds to
// an even and to an odd pattern; they differ by one at most (fl does not change the order of two sums, and two
// that have become equally even stay in step), and two stretches make one. A stretch of lanes whose
// binade is certain is one such pair (kind RUN; Units in molla_exact.cuh). A lane near the end of a binade carries
// the pairs of both binades (DUAL); a lane that outgrows a binade by itself or whose
// guess spans more is added value by value (STEP). The binades are guessed from the estimated
// sum before the tile; whoever runs the items checks every guess against the exact sum and adds the
// values one by one where it was wrong.
enum { K_RUN = 0, K_DUAL = 1, K_STEP = 2 };
struct __align__(16) Item {
    unsigned int ka, kb;   // units of binade jb (RUN, DUAL) and of the next one (DUAL), see units()
    unsigned int meta;     // biased exponent of the binade (8 bits), kind (2), place of the values (8; 255: the list), tile (10)
    unsigned int oc;       // entries (11 bits), first entry in the tile's list (10), number of the item in its tile (7)
    __device__ __forceinline__ unsigned int jb() const { return meta & 0xffu; }
    __device__ __forceinline__ unsigned int kind() const { return (meta >> 8) & 3u; }
    __device__ __forceinline__ unsigned int place() const { return (meta >> 10) & 0xffu; }
    __device__ __forceinline__ int tile() const { return (int)(meta >> 18); }
    __device__ __forceinline__ int cnt() const { return (int)(oc & 0x7ffu); }
    __device__ __forceinline__ int off() const { return (int)((oc >> 11) & 0x3ffu); }
    __device__ __forceinline__ int num() const { return (int)(oc >> 21); }
};
// ---- settings ---------------------------------------------------------------------------------
struct __align__(16) RowCfg {
    long long lrow;
    float T, P, minp, typ, rp, fp, pp;
    int q, k, ring_n, H, b0, nb, npatch;
    const long long *histp;
    long long n_lim;
    bool greedy, topp_on, pure, open_row;
    bool late;              // the row is looked at again once it is answered (F_JUMP): its state moves on behind that
    unsigned int status;
};

// What row_plan hands to the kernels behind it.
struct __align__(16) RowPlan { RowCfg c; int kind, flags; float top; unsigned int tau_bits; float xmax; int imax; int need; unsigned int tau_far; };

// A row's small results, together in memory: the kernels that read them wait once.
//   RowHead | TileOut[ntile] | candidates[HEADCAP] | prefix sums[HEADCAP] | values of careful chunks[CARE_PLACES][32] | items
// A walk past the head: per binade of the running sum, the integer mass of every bin of values, and the
// elements that would round on a tie there.
constexpr int WALK_BINADES = 3;
struct __align__(16) WalkTies { int n; int pad[3]; unsigned long long key[TIE_CAP]; };
// The bins whose elements the walk will want one by one, and those elements.
constexpr int PICKS = 8, PICK_CAP = NC;
struct __align__(16) WalkPicks { int n, arrived, pad[2]; int bin[PICKS]; int cnt[PICKS]; };
constexpr size_t WALK_BYTES = WALK_BINADES * (NBINS * sizeof(unsigned long long) + sizeof(WalkTies)) + sizeof(WalkPicks) + (size_t)PICKS * PICK_CAP * sizeof(unsigned long long);

struct __align__(16) RowHead { RowPlan plan; int ncand, nitem, ncare, state; float Z, head_s; long long head_pos; unsigned int hits[4]; int nfar, pad[3]; };   // hits: see F_JUMP

struct RowsArgs {
    BatchArgs a;
    int r0, rows;            // batch rows [r0, r0 + rows) are in flight
    int ntile, nspan;
    int oG, oVc, oL;         // see F_NARROW
    bool late_next;          // row_tail lets the next kernel begin once it has begun itself, not before
    int need_far, need_topk; // lanes' maxima that reach a far head's edge, without a top-k and with one; 0: rows of this length have none
    TileStat *ts;            // [rows][ntile]
    float *gmax;             // [rows][ntile * 32] the lanes' maxima
    TilePlan *tp;            // [rows][ntile]
    char *box; long long box_stride;  // [rows]
    int *queue;              // rows for tile_walk and row_tail: their number, then the rows
    char *walk;              // [rows] tables and ties of a walk past the head
    float *elist;            // [rows][ntile][TILE] values kept, in vocabulary order, packed per tile
    unsigned int *kmask;     // [rows][ntile][32] which logits they are
    __device__ __forceinline__ unsigned long long *table(int rr, int b) const { return reinterpret_cast<unsigned long long *>(walk + (size_t)rr * WALK_BYTES) + (size_t)b * NBINS; }
    __device__ __forceinline__ WalkTies *ties(int rr) const { return reinterpret_cast<WalkTies *>(table(rr, WALK_BINADES)); }
    __device__ __forceinline__ WalkPicks *picks(int rr) const { return reinterpret_cast<WalkPicks *>(ties(rr) + WALK_BINADES); }
    __device__ __forceinline__ unsigned long long *picked(int rr, int i) const { return reinterpret_cast<unsigned long long *>(picks(rr) + 1) + (size_t)i * PICK_CAP; }
    __device__ __forceinline__ unsigned long long *far(int rr) const { return picked(rr, 0); }   // (row_head has read it before tile_pick writes there)
    __device__ __forceinline__ RowHead *head(int rr) const { return reinterpret_cast<RowHead *>(box + (long long)rr * box_stride); }
    __device__ __forceinline__ TileOut *to(int rr) const { return reinterpret_cast<TileOut *>(head(rr) + 1); }
    __device__ __forceinline__ unsigned long long *cand(int rr) const { return reinterpret_cast<unsigned long long *>(to(rr) + ((ntile + 1) & ~1)); }
    __device__ __forceinline__ float *pre(int rr) const { return reinterpret_cast<float *>(cand(rr) + HEADCAP); }
    __device__ __forceinline__ float *care(int rr) const { return pre(rr) + HEADCAP; }
    __device__ __forceinline__ Item *items(int rr) const { return reinterpret_cast<Item *>(care(rr) + CARE_PLACES * 32); }
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Where row r's settings live and what they are; status bits for a row that cannot be sampled
// (the rules of SamplerConfig.check, sample.mojo:140-154; NaN fails every test).
__device__ __forceinline__ RowCfg row_cfg(const BatchArgs &a, int r) {
    RowCfg c;
    c.status = 0;
    c.late = false;
    c.q = a.slot ? a.slot[r] : r;
    c.lrow = a.rows ? (long long)a.rows[r] : (long long)r;
    const bool idx_ok = (!a.slot || (c.q >= 0 && (a.n_slots <= 0 || c.q < a.n_slots))) &&
                        (!a.rows || (c.lrow >= 0 && (a.n_logit_rows <= 0 || c.lrow < a.n_logit_rows)));
    const int q = idx_ok ? c.q : 0;   // a stale row or slot index: nothing of that row or slot is touched
    if (!idx_ok) {
        c.T = 0; c.P = 1; c.minp = 0; c.typ = 1; c.rp = 1; c.fp = c.pp = 0; c.k = 0; c.ring_n = c.H = c.b0 = c.nb = c.npatch = 0;
        c.histp = nullptr; c.n_lim = a.V; c.greedy = true; c.topp_on = c.pure = c.open_row = false;
        c.status = MOLLA_ROW_INVALID_CONFIG | 0x80000000u;
        return c;
    }
    c.T = a.temperature ? a.temperature[q] : 0.0f;
    c.k = a.top_k ? a.top_k[q] : 0;
    c.P = a.top_p ? a.top_p[q] : 1.0f;
    c.minp = a.min_p ? a.min_p[q] : 0.0f;
    c.typ = a.typical_p ? a.typical_p[q] : 1.0f;
    c.rp = a.repeat_penalty ? a.repeat_penalty[q] : 1.0f;
    c.fp = a.frequency_penalty ? a.frequency_penalty[q] : 0.0f;
    c.pp = a.presence_penalty ? a.presence_penalty[q] : 0.0f;
    c.ring_n = a.ring ? min(max(a.ring_len[q], 0), a.ring_cap) : 0;
    const bool won = a.ring ? (c.ring_n > 0) : (a.window_on ? (a.window_on[q] != 0) : true);
    const int h0 = (a.hist && a.hist_off) ? a.hist_off[q] : 0;
    // a window kept on the device fills from its first slot (sample.mojo:246-258): the first
    // `filled` entries are the window, whatever the head is
    c.histp = a.ring ? a.ring + (size_t)q * (size_t)a.ring_cap : (a.hist ? a.hist + h0 : nullptr);
    c.H = a.ring ? min(max(a.ring_filled[q], 0), c.ring_n) : ((a.hist && a.hist_off) ? (a.hist_off[q + 1] - h0) : 0);
    c.b0 = (a.bias_ids && a.bias_off) ? a.bias_off[q] : 0;
    c.nb = (a.bias_ids && a.bias_off) ? (a.bias_off[q + 1] - c.b0) : 0;
    const bool valid = (c.T >= 0.0f) && (c.k >= 0) && (c.P > 0.0f && c.P <= 1.0f) && (c.minp >= 0.0f && c.minp <= 1.0f) &&
                       (c.typ > 0.0f && c.typ <= 1.0f) && (c.rp > 0.0f) && c.H >= 0 && c.nb >= 0;
    c.greedy = !(c.T > 0.0f);
    const bool penalizing = won && c.H > 0 && (c.rp != 1.0f || c.fp != 0.0f || c.pp != 0.0f);
    c.npatch = (penalizing ? c.H : 0) + c.nb;
    if (!valid) c.status |= MOLLA_ROW_INVALID_CONFIG;
    // typical-p is done on rows an earlier filter sorted and cut to a set inside the sorted head
    else if (!c.greedy && c.typ < 1.0f && !((c.k > 0 && c.k < a.V) || c.P < 1.0f)) c.status |= MOLLA_ROW_UNSUPPORTED;
    if (c.npatch > PATCH_MAX) c.status |= MOLLA_ROW_UNSUPPORTED;
    c.n_lim = (c.k > 0 && c.k < a.V) ? (long long)c.k : (long long)a.V;
    c.open_row = c.n_lim == (long long)a.V;
    c.topp_on = c.P < 1.0f && c.n_lim > 1;
    c.pure = !c.topp_on && c.open_row;
    return c;
}

// `_took` (sample.mojo:361-363), one thread: the picked token into the slot's window, the draw counter on.
__device__ __forceinline__ void took_row(const BatchArgs &a, int r, const RowCfg &c, int token) {
    if (!a.ring || token < 0) return;
    // (all loads before the stores: one round trip instead of four)
    const bool seen = c.ring_n > 0;
    const int q = c.q, hd = seen ? a.ring_head[q] : 0, f = seen ? a.ring_filled[q] : 0;
    const unsigned long long dn = a.drawn_rw[q];
    const long long stop = a.stopped && a.stop_token ? a.stop_token[q] : -1ll;
    if (seen) {  // `observe` (:246-258)
        const int at = (hd >= 0 && hd < c.ring_n) ? hd : 0;
        a.ring[(size_t)q * (size_t)a.ring_cap + at] = (long long)token;
        a.ring_head[q] = (at + 1) % c.ring_n;
        a.ring_filled[q] = f < c.ring_n ? f + 1 : c.ring_n;
    }
    a.drawn_rw[q] = dn + 1ull;
    if (a.stopped) a.stopped[r] = (a.stop_token && stop == (long long)token) ? 1 : 0;
}

// A row's answer, one thread; returns the token, -1 where there is none.
__device__ __forceinline__ int answer_row(const BatchArgs &a, int r, unsigned int status, int token, float dZ, float dsum, float dtarget, float dp) {
    if (status & 0x80000000u) {  // a stale index
        a.tokens[r] = -1; a.row_status[r] = status & 0x7fffffffu;
        return -1;
    }
    if (status & (MOLLA_ROW_LOAD_TIMEOUT | MOLLA_ROW_DEGENERATE | MOLLA_ROW_INVALID_CONFIG | MOLLA_ROW_UNSUPPORTED | MOLLA_ROW_EMPTY)) token = -1;
    a.tokens[r] = token;
    a.row_status[r] = status;
    if (a.diag) { a.diag[4 * r] = dZ; a.diag[4 * r + 1] = dsum; a.diag[4 * r + 2] = dtarget; a.diag[4 * r + 3] = dp; }
    return token;
}

// The end of a row, one thread: the answer, then `_took`.
__device__ __noinline__ void finish_row(const BatchArgs &a, int r, const RowCfg &c, unsigned int status, int token, float dZ, float dsum,
                           float dtarget, float dp) {
    token = answer_row(a, r, status, token, dZ, dsum, dtarget, dp);
    if (!c.late) took_row(a, r, c, token);
}

// ---- arithmetic -------------------------------------------------------------------------------
// (out of line: the compiler's division is long, and a row's code is read from L2 once per SM)
__device__ __noinline__ float div_slow(float x, float d) { return __fdiv_rn(x, d); }
// a probability e / Z (Z between 1 and the vocabulary's size; e in [0, 1])
__device__ __forceinline__ float prob_of(float e, float Z, float y) {
    return e > 1.0e-20f || e == 0.0f ? div_by(e, Z, y) : div_slow(e, Z);
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_max_key(float v) { return fkey_inv(__reduce_max_sync(0xffffffffu, fkey(v))); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---- a span of a row in shared memory -----------------------------------------------------------
__device__ __forceinline__ void cp16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct SpanScratch {
    unsigned int cnt[SPAN / 2];         // per logit 16 bits: times in the window, top bit: named by a bias
    unsigned short hits[PATCH_MAX];     // the patched logits of the span
    int nhits;
};

// Logits [c0, c0 + SPAN) of logit row `lrow` on their way to `sx`: lane l of tile w will find its 32 at
// sx[(32 w + l) * PITCH]. What lies past the row's end is -inf. 16-byte asynchronous copies where the row
// starts on such a boundary, 4-byte ones elsewhere.
__device__ __forceinline__ void span_fetch(const BatchArgs &a, long long lrow, int c0, float *sx) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *src = a.logits + lrow * a.row_stride + c0;
    const int n = min(SPAN, a.V - c0), e0 = warp * TILE;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0 && e0 + TILE <= n) {
        float *dst = sx + (warp * 32 + (lane >> 3)) * PITCH + (lane & 7) * 4;
        const float *from = src + e0 + lane * 4;
#pragma unroll
        for (int i = 0; i < 8; i++) cp16(dst + i * 4 * PITCH, from + i * 128);
    } else {
#pragma unroll 4
        for (int i = 0; i < 32; i++) {
            const int e = e0 + i * 32 + lane;
            float *dst = sx + (warp * 32 + i) * PITCH + lane;
            if (e < n) cp4(dst, src + e);
            else *dst = -INFINITY;
        }
    }
}

// Waits for what span_fetch asked for and caps, masks, biases and penalises it. Threads
// 0..SPAN_THREADS-1 work (`active`), all threads of the block take part in the barriers; each warp may
// then use its own tile.
__device__ void span_ready(const BatchArgs &a, const RowCfg &c, int r, int c0, float *sx, SpanScratch *s, bool active, bool mine_on = true) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = min(SPAN, a.V - c0);
    const int e0 = warp * TILE;
    float *mine = sx + (size_t)tid * PITCH;
    const bool patching = c.npatch > 0;
    if (patching) {
        if (active) {
            uint4 *z = reinterpret_cast<uint4 *>(s->cnt);
#pragma unroll
            for (int i = 0; i < SPAN / 8 / SPAN_THREADS; i++) z[tid + i * SPAN_THREADS] = make_uint4(0, 0, 0, 0);
            if (tid == 0) s->nhits = 0;
        }
        __syncthreads();
        if (active)
#pragma unroll 1
            for (int i = tid; i < c.npatch; i += SPAN_THREADS) {
                const bool is_bias = i < c.nb;
                const long long t64 = (is_bias ? a.bias_ids[c.b0 + i] : c.histp[i - c.nb]) - (long long)c0;
                if (t64 < 0 || t64 >= n) continue;
                const int t = (int)t64, sh = (t & 1) * 16;
                const unsigned int old = is_bias ? atomicOr(&s->cnt[t >> 1], 0x8000u << sh) : atomicAdd(&s->cnt[t >> 1], 1u << sh);
                if (((old >> sh) & 0xffffu) == 0u) s->hits[satom_add(&s->nhits, 1)] = (unsigned short)t;
            }
        __syncthreads();
    }
    if (active) {
        cp_wait();
        __syncwarp();
        const int m = mine_on ? n - (e0 + lane * 32) : 0;  // this lane's logits that exist
        if (a.softcap > 0.0f) {
            const float rcap = softcap_plain(a.softcap) ? __frcp_rn(a.softcap) : 0.0f;
#pragma unroll 1
            for (int j = 0; j < min(32, m); j += 4) {   // (what lies past the row's end stays -inf)
                float4 &v = *reinterpret_cast<float4 *>(mine + j);
                float x[4] = {v.x, v.y, v.z, v.w};
                softcap4(x, a.softcap, rcap);
                v = make_float4(x[0], j + 1 < m ? x[1] : -INFINITY, j + 2 < m ? x[2] : -INFINITY, j + 3 < m ? x[3] : -INFINITY);
            }
            __syncwarp();
        }
        if (a.mask && m > 0) {
            // `_mask` (sample.mojo:371-379): what the grammar forbids is no candidate at all. A logit of
            // -inf is exactly that here: it wins no maximum, no bias or penalty brings it back, its
            // exponential is zero, and zeros are absent from every sum, count and walk.
            const unsigned int w = __ldg(a.mask + (long long)r * a.mask_stride + ((c0 + e0 + lane * 32) >> 5));
#pragma unroll
            for (int g = 0; g < 8; g++) {
                float4 x = *reinterpret_cast<float4 *>(mine + 4 * g);
                if (!((w >> (4 * g)) & 1u)) x.x = -INFINITY;
                if (!((w >> (4 * g + 1)) & 1u)) x.y = -INFINITY;
                if (!((w >> (4 * g + 2)) & 1u)) x.z = -INFINITY;
                if (!((w >> (4 * g + 3)) & 1u)) x.w = -INFINITY;
                *reinterpret_cast<float4 *>(mine + 4 * g) = x;
            }
        }
    }
    if (patching) {
        __syncthreads();
        if (active) {
            const int nh = s->nhits;
#pragma unroll 1
            for (int i = tid; i < nh; i += SPAN_THREADS) {
                const int t = s->hits[i];
                const int nw = (int)((s->cnt[t >> 1] >> ((t & 1) * 16)) & 0x7fffu);
                float v = sx[(t >> 5) * PITCH + (t & 31)];
#pragma unroll 1
                for (int b = 0; b < c.nb; b++)  // duplicates add up, in the order they were given
                    if (a.bias_ids[c.b0 + b] == (long long)t + c0) v = __fadd_rn(v, a.bias_vals[c.b0 + b]);
                if (nw > 0) {
                    if (v > 0.0f) v = __fdiv_rn(v, c.rp);
                    else v = __fmul_rn(v, c.rp);
                    v = __fsub_rn(v, __fmul_rn((float)nw, c.fp));
                    v = __fsub_rn(v, c.pp);
                }
                sx[(t >> 5) * PITCH + (t & 31)] = v;
            }
        }
        __syncthreads();
    } else {
        __syncwarp();
    }
}

// =============================================================================
// Kernel 1: the tiles' maxima and estimated sums. Bound: HBM (4 bytes per logit, once): 156 MB take 43 us
// (3.6 TB/s), 537 MB 98 us (5.5 TB/s). A warp has its tile in shared memory by asynchronous copies,
// four blocks of 8192 logits an SM in flight; a tile per warp, because then nothing but a warp waits for
// it, and of 1024 logits, because a lane's 32 are what the items' chunks are made of.
// =============================================================================
struct SpanShared {
    float x[SPAN_THREADS * PITCH];
    SpanScratch s;
};

__global__ void __launch_bounds__(SPAN_THREADS, 4) tile_stats_kernel(const __grid_constant__ RowsArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SpanShared *S = reinterpret_cast<SpanShared *>(smem_raw);
    pdl_next();
    pdl_wait();
    const int rr = blockIdx.x / A.nspan, span = blockIdx.x - rr * A.nspan, r = A.r0 + rr;
    const BatchArgs &a = A.a;
    {   // the logits first: what the settings say about them can wait
        const long long lrow = a.rows ? (long long)a.rows[r] : (long long)r;
        if (lrow >= 0 && (!a.rows || a.n_logit_rows <= 0 || lrow < a.n_logit_rows)) span_fetch(a, lrow, span * SPAN, S->x);
    }
    const RowCfg c = row_cfg(a, r);
    if (c.status) { cp_wait(); return; }
    span_ready(a, c, r, span * SPAN, S->x, &S->s, true);
    const int lane = threadIdx.x & 31, tile = span * (SPAN / TILE) + (threadIdx.x >> 5);
    if (tile >= A.ntile) return;
    const float *mine = S->x + threadIdx.x * PITCH;
    float x[32];
#pragma unroll
    for (int g = 0; g < 8; g++) {
        const float4 v = *reinterpret_cast<const float4 *>(mine + 4 * g);
        x[4 * g] = v.x; x[4 * g + 1] = v.y; x[4 * g + 2] = v.z; x[4 * g + 3] = v.w;
    }
    float m = x[0];
#pragma unroll
    for (int j = 1; j < 32; j++) m = fmaxf(m, x[j]);
    const float tmax = warp_max_key(m);
    const unsigned int who = __ballot_sync(0xffffffffu, m == tmax);
    const int first = who ? __ffs((int)who) - 1 : 0;   // the first line that holds the maximum, and where in it (a lane looks at a logit)
    const unsigned int where = __ballot_sync(0xffffffffu, S->x[((threadIdx.x & ~31) + first) * PITCH + lane] == tmax);
    const int at = (where ? __ffs((int)where) - 1 : 0) + first * 32 + tile * TILE;
    const bool sampled = !c.greedy && c.n_lim > 1;
    int eq = 0;
    float sum = 0.0f;
    if (sampled) {
        // an estimate is enough (it only guesses binades and bounds what is dropped): hardware exponentials
        if (tmax > -INFINITY) {
            const float f = fminf(1.44269504f / c.T, 1.0e30f);
            float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                s0 += ex2_approx((x[j] - tmax) * f);
                s1 += ex2_approx((x[j + 1] - tmax) * f);
            }
            sum = warp_sum(s0 + s1);
        }
        A.gmax[((size_t)rr * A.ntile + tile) * 32 + lane] = m;
    } else if (!c.greedy) {  // only a top-k of one asks how many share the maximum
#pragma unroll
        for (int j = 0; j < 32; j++) eq += x[j] == tmax ? 1 : 0;
        eq = __reduce_add_sync(0xffffffffu, eq);
    }
    if (lane == 0) {
        TileStat t;
        t.tmax = tmax; t.tsum = sum; t.tidx = at; t.teq = eq;
        A.ts[(size_t)rr * A.ntile + tile] = t;
    }
}

// =============================================================================
// Kernel 2: one block per row. Bound: latency (two rounds of loads, one histogram, code that runs once):
// 5 us for 128 greedy rows, 9 for 64 sampled ones, 14 for 256, 21 for 512. The settings are stored as soon as the row
// is known to be sampled: kept in registers to the end they spilled, and 512 rows took 3 us more.
// =============================================================================
struct JumpShared { float in[128], over[128], own[128]; unsigned int hits[4]; };
struct PlanShared {
    union { unsigned int hist[PLAN_BINS]; JumpShared jump; };
    int edge, edge_far;
    float wsf[NWARP + 1];
    int wsi[NWARP + 1];
};

// Exclusive scan over the block without a subtraction (the terms span many orders of magnitude).
__device__ __forceinline__ float block_excl_scan_plus(float v, float *ws, float *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float inc = warp_incl_scan(v, lane);
    float ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = 0.0f;
    __syncthreads();
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    float b = 0.0f, t = 0.0f;
#pragma unroll
    for (int w = 0; w < NWARP; w++) {
        if (w == warp) b = t;
        t += ws[w];
    }
    *total = t;
    return b + ex;
}

// Rows whose running sum jumps: MOLLA_ROW_SLOW_PATH tells a caller that the guesses of the sum's binade
// went wrong somewhere. They are made for ranges of oL logits, 32 ranges to a group, with a prefix over
// the groups of a block that is taken by subtracting a group's own sum, in double precision; where that
// sum is more than 2^40 times everything before it, too few bits are left of what came before. This finds the
// groups where that may be: the estimated sum of their tiles
// against the largest term before them. Only sharp rows (low temperatures) have one.
// Block of NT threads, 4 to a group; bit q of J.hits is set for group q (block q / 16 of the layout, warp q % 16).
__device__ __noinline__ bool find_jumps(const RowsArgs &A, int rr, float f, float xmax, JumpShared &J) {
    const int tid = threadIdx.x, lane = tid & 31, q = tid >> 2, part = tid & 3, g = q >> 4, w = q & 15, V = A.a.V;
    const float *gm = A.gmax + (size_t)rr * A.ntile * 32;
    const int e = min(V, (g + 1) * A.oVc), a = min(e, g * A.oVc + w * 32 * A.oL), b = min(e, a + 32 * A.oL);
    float in = -INFINITY, over = -INFINITY;
    if (g < A.oG && b > a) {
#pragma unroll 8
        for (int k = (a >> 5) + part; k <= (b - 1) >> 5; k += 4) {
            const float m = gm[k];
            over = fmaxf(over, m);
            if (k * 32 >= a && k * 32 + 32 <= b) in = fmaxf(in, m);
        }
    }
    in = fmaxf(in, __shfl_xor_sync(0xffffffffu, in, 1)); over = fmaxf(over, __shfl_xor_sync(0xffffffffu, over, 1));
    in = fmaxf(in, __shfl_xor_sync(0xffffffffu, in, 2)); over = fmaxf(over, __shfl_xor_sync(0xffffffffu, over, 2));
    __syncthreads();
    if (part == 0) {
        float own = 0.0f;
        if (over > -INFINITY)
#pragma unroll 4
            for (int t = a / TILE; t <= (b - 1) / TILE; t++) {
                const TileStat st = A.ts[(size_t)rr * A.ntile + t];
                if (st.tmax > over) {   // (a tile that reaches out of the group: its lanes' maxima bound what is inside)
#pragma unroll 8
                    for (int k = max(t * 32, a >> 5); k < min(t * 32 + 32, ((b - 1) >> 5) + 1); k++) own += 32.0f * ex2_approx(fminf((gm[k] - over) * f, 0.0f));
                } else if (st.tmax > -INFINITY) own += st.tsum * ex2_approx((st.tmax - over) * f);
            }
        J.in[q] = in; J.over[q] = over; J.own[q] = log2f(fminf(own, (float)(b - a)));
    }
    __syncthreads();
    bool any = false;
    if (tid < 128) {
        float pf = lane > 0 ? J.in[tid - 1] : -INFINITY;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float v = __shfl_up_sync(0xffffffffu, pf, o); if (lane >= o) pf = fmaxf(pf, v); }
#pragma unroll 4
        for (int i = 0; i < (tid & ~31); i++) pf = fmaxf(pf, J.in[i]);
        // (e^-105 and less is zero)
        any = (tid & 15) != 0 && J.over[tid] > -INFINITY && pf > -INFINITY && (J.over[tid] - pf) * f + J.own[tid] > 39.9f && (xmax - pf) * f < 152.0f;
        const unsigned int m = __ballot_sync(0xffffffffu, any);
        if (lane == 0) J.hits[tid >> 5] = m;
    }
    return __syncthreads_or(any) != 0;
}

// (the settings as soon as the row is known to be sampled: they are not kept in registers to the end)
__device__ __forceinline__ void store_settings(const RowsArgs &A, int rr, const RowCfg &c) {
    RowHead *h = A.head(rr);
    h->plan.c = c;
    h->ncand = 0; h->nfar = 0; h->nitem = 0; h->ncare = 0; h->state = 0;
    if (rr == 0) A.queue[0] = 0;
}
__device__ __forceinline__ void store_done(const RowsArgs &A, int rr) {   // (nothing else of such a row is looked at)
    A.head(rr)->plan.kind = PLAN_DONE;
    if (rr == 0) A.queue[0] = 0;
}

__global__ void __launch_bounds__(NT) row_plan_kernel(const __grid_constant__ RowsArgs A) {
    __shared__ PlanShared S;
    pdl_next();
    const int rr = blockIdx.x, r = A.r0 + rr, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const BatchArgs &a = A.a;
    pdl_wait();
    RowCfg c = row_cfg(a, r);
    if (MOLLA_KNOB(a, 16) && !c.status) c.status |= MOLLA_ROW_LOAD_TIMEOUT;  // testing build: a wait that ran out
    if (c.status) {
        if (tid == 0) { answer_row(a, r, c.status, -1, 0, 0, 0, 0); store_done(A, rr); }
        return;
    }
    // the maximum and its first index (kernel.mojo:571-585, sample.mojo:342-346)
    const TileStat *ts = A.ts + (size_t)rr * A.ntile;
    float tm[2], tsum[2], xmax = -INFINITY;
    int te[2], imax = 0x7fffffff;
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int t = 2 * tid + u;
        TileStat s;
        s.tmax = -INFINITY; s.tsum = 0.0f; s.tidx = 0x7fffffff; s.teq = 0;
        if (t < A.ntile) s = ts[t];
        tm[u] = s.tmax; tsum[u] = s.tsum; te[u] = s.teq;
        if (s.tmax > xmax) { xmax = s.tmax; imax = s.tidx; }
    }
    warp_argmax(xmax, imax);
    if (lane == 0) { S.wsf[warp] = xmax; S.wsi[warp] = imax; }
    __syncthreads();
    xmax = S.wsf[0]; imax = S.wsi[0];
#pragma unroll
    for (int w = 1; w < NWARP; w++)
        if (S.wsf[w] > xmax || (S.wsf[w] == xmax && S.wsi[w] < imax)) { xmax = S.wsf[w]; imax = S.wsi[w]; }
    if (imax == 0x7fffffff) imax = 0;
    unsigned int status = 0;
    bool done = c.greedy || c.n_lim == 1;
    if (a.mask && !(xmax > -INFINITY)) { status |= MOLLA_ROW_EMPTY; done = true; }  // every candidate was filtered out
    else if (!c.greedy && c.n_lim == 1) {
        // top-k of one: the sort's first element is a maximum (sample.mojo:485-490)
        int eq = 0;
#pragma unroll
        for (int u = 0; u < 2; u++) eq += tm[u] == xmax ? te[u] : 0;
        eq = __reduce_add_sync(0xffffffffu, eq);
        __syncthreads();
        if (lane == 0) S.wsi[warp] = eq;
        __syncthreads();
        eq = 0;
        for (int w = 0; w < NWARP; w++) eq += S.wsi[w];
        if (eq > 1) status |= MOLLA_ROW_TOPK_TIE;
    }
    if (done) {
        if (tid == 0) { took_row(a, r, c, answer_row(a, r, status, imax, 0, 0, 0, 0)); store_done(A, rr); }
        return;
    }
    if (tid == 0) store_settings(A, rr, c);
    const float top = (c.T == 1.0f) ? xmax : __fdiv_rn(xmax, c.T);
    const bool filter_ok = fabsf(top) < 1.0e5f;
    long long need = c.open_row ? (long long)HEAD_NEED : c.n_lim + 1;
    if (need > HEAD_MOST) need = HEAD_MOST;
    if (need > a.V) need = a.V;
    // estimated sum before every tile, relative to the row's maximum
    const float f = fminf(1.44269504f / c.T, 1.0e30f);
    float e[2];
#pragma unroll
    for (int u = 0; u < 2; u++) e[u] = (tm[u] > -INFINITY) ? tsum[u] * ex2_approx((tm[u] - xmax) * f) : 0.0f;
    const float first = A.gmax[(size_t)rr * A.ntile * 32];   // of the first 32 logits
    float total;
    const float ex = block_excl_scan_plus(e[0] + e[1], S.wsf, &total);
    const float est[2] = {ex, ex + e[0]};
    // A logit below half an ulp of the running sum adds nothing to it, whatever order: 17.6 is above
    // 25 ln 2, the tenth taken off the estimate covers what rounding loses. Below top - 105 the
    // exponential is exactly zero.
    const float thr_zero = filter_ok ? c.T * (top - 105.0f) : -INFINITY;
    auto thr_of = [&](float s) -> float {
        const float rel = (filter_ok && s > 0.0f) ? c.T * (top + logf(0.9f * s) - REL_MARGIN) : -INFINITY;
        return fmaxf(rel, thr_zero);
    };
    // The head: a value that at least `need` of the lanes' maxima reach bounds the need-th largest
    // element from below, and few more elements than that reach it.
    float tau_x = INFINITY, far_x = INFINITY;
    bool narrow = false, far = false;
    if (!c.pure) {
        const int ng = A.ntile * 32;
        const float *gm = A.gmax + (size_t)rr * ng;
        // one histogram of the lanes' maxima by distance below the row's
#pragma unroll 1
        for (int i = tid; i < PLAN_BINS; i += NT) S.hist[i] = 0u;
        if (tid == 0) S.edge = S.edge_far = -1;
        __syncthreads();
#pragma unroll 1
        for (int i0 = 0; i0 < ng; i0 += 8 * NT) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = (i0 + u * NT + tid < ng) ? gm[i0 + u * NT + tid] : -INFINITY;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const float d = (xmax - v[u]) * PLAN_RES;
                if (d < (float)PLAN_BINS) sred_add(&S.hist[(int)d], 1u);
            }
        }
        __syncthreads();
        constexpr int PER = PLAN_BINS / NT;
        int n[PER], sum = 0, tot;
#pragma unroll
        for (int i = 0; i < PER; i++) { n[i] = (int)S.hist[PER * tid + i]; sum += n[i]; }
        int run = block_excl_scan<int>(sum, S.wsi, &tot);
        // (typical-p works on what the near head holds, and refuses more)
        const int need_far = A.need_far == 0 ? 0 : (c.open_row ? (c.topp_on && !(c.typ < 1.0f) ? min(A.need_far, tot) : 0) : min(A.need_topk, tot));
#pragma unroll
        for (int i = 0; i < PER; i++) {
            if (run < need && run + n[i] >= need) S.edge = PER * tid + i;
            if (run < need_far && run + n[i] >= need_far) S.edge_far = PER * tid + i;
            run += n[i];
        }
        __syncthreads();
        // (a bin's lower end, and a little below it: the subtraction and the product above were rounded)
        auto below_bin = [&](int b) { return fabsf(xmax) < 65536.0f ? xmax - ((float)(b + 1) + 0.25f) * (1.0f / PLAN_RES) : -INFINITY; };
        tau_x = S.edge >= 0 ? below_bin(S.edge) : -INFINITY;
        // (what cannot matter to the whole sum is no use to an open row's head: a sharp row has few elements that can)
        far_x = S.edge_far >= 0 ? fmaxf(below_bin(S.edge_far), c.open_row ? thr_of(total) : -INFINITY) : -INFINITY;
        far = far_x > -INFINITY && (c.open_row ? far_x < (tau_x > -INFINITY ? tau_x : INFINITY) : far_x > tau_x);
        // F_NARROW: a top-k so wide for the vocabulary that fewer ranges than candidates exist (one range
        // per thread of the widest layout: oG blocks of NT threads with oL logits each). Such rows report
        // the order of equal probabilities the way the descending walk sees it.
        if (need > HEAD_NEED && A.oG > 0) {
            int have = 0, allowed = 0;
#pragma unroll 1
            for (int i = tid; i < A.oG * NT; i += NT) {
                const int g = i / NT, l0 = (i - g * NT) * A.oL, n_g = max(0, min(A.oVc, a.V - g * A.oVc));
                if (l0 >= n_g) continue;
                int bits = min(A.oL, n_g - l0);
                if (a.mask) {
                    const unsigned int *mrow = a.mask + (long long)r * a.mask_stride;
                    int b = 0;
#pragma unroll 1
                    for (int j = 0; j < bits; j++) { const int t = g * A.oVc + l0 + j; b += (__ldg(mrow + (t >> 5)) >> (t & 31)) & 1u; }
                    bits = b;
                }
                have += bits > 0 ? 1 : 0;
                allowed += bits;
            }
            have = __reduce_add_sync(0xffffffffu, have);
            allowed = __reduce_add_sync(0xffffffffu, allowed);
            if (lane == 0) { S.wsi[warp] = have; S.wsf[warp] = __int_as_float(allowed); }
            __syncthreads();
            have = allowed = 0;
            for (int w = 0; w < NWARP; w++) { have += S.wsi[w]; allowed += __float_as_int(S.wsf[w]); }
            narrow = have < need && allowed > HEADCAP;
            __syncthreads();
        }
    }
    bool jump = false;
    if (A.oG > 0 && !((xmax - first) * f <= 29.0f)) {
        __syncthreads();
        jump = find_jumps(A, rr, f, xmax, S.jump);
        if (jump && tid < 4) A.head(rr)->hits[tid] = S.jump.hits[tid];
    }
    auto bits_of = [&](float x) -> unsigned int {
        const unsigned int b = __float_as_uint(expf_pinned(__fsub_rn((c.T == 1.0f) ? x : __fdiv_rn(x, c.T), top)));
        return b > 5u ? b - 4u : 1u;
    };
    const float keep_x = far && far_x < tau_x ? far_x : tau_x;
    TilePlan *tp = A.tp + (size_t)rr * A.ntile;
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int t = 2 * tid + u;
        if (t < A.ntile) { TilePlan p; p.thr = fminf(thr_of(est[u]), keep_x); p.est = est[u]; tp[t] = p; }
    }
    if (tid == 0) {
        RowPlan &pl = A.head(rr)->plan;
        pl.kind = PLAN_SAMPLED;
        const bool past_head = c.n_lim + 1 > (c.open_row ? HEAD_NEED : HEAD_MOST);
        // (too few lanes to bound the head: row_finish narrows it down from the list)
        pl.flags = ((c.pure || past_head || !(tau_x > -INFINITY)) ? F_LIST : 0) | (c.pure ? F_PURE : 0) | (narrow ? F_NARROW : 0) | (jump ? F_JUMP : 0) |
                   (far ? F_FAR | (c.open_row && tau_x > -INFINITY ? 0 : F_ALLNEAR) : 0) | ((filter_ok && fabsf(top) > 1.0e-6f && c.T > 1.0e-9f && c.T < 1.0e9f) ? F_FASTDIV : 0);
        if (jump) pl.c.late = true;
        pl.top = top; pl.tau_bits = c.pure ? 0xffffffffu : bits_of(tau_x);
        pl.tau_far = far ? bits_of(far_x) : pl.tau_bits;
        pl.xmax = xmax; pl.imax = imax; pl.need = (int)need;
    }
}

// =============================================================================
// Kernel 3: exponentials, candidates, items. Bound: instructions, and the latency of the plan's and the tile's loads:
// about 1000 warp instructions a tile of a row whose list nobody wants (near_units), 2300 where it is wanted and two
// thirds are kept. 256 rows of 151936, mixed, take 64 us (all evaluated in full and every tile cut into chunks: 74),
// 512 of 262144 with a top-k of 1024 200 (245), issuing in 60 % of the active cycles. Evaluating in full warps from
// a list of what is kept, in place of each lane its own, gave 20 %.
// =============================================================================
// A tile's list in shared memory: entry e at list[skew(e)] (a word is left out after every 32, so that
// lanes that read their own chunks meet different banks). Lane l's chunk is entries [off, off + cnt):
// equal shares of an odd number, or 32.
__device__ __forceinline__ int skew(int e) { return e + (e >> 5); }
struct TileChunk { int cnt, off, total; float csum; };
__device__ __forceinline__ TileChunk tile_chunk(const float *list, int total) {
    TileChunk c;
    int per = (total + 31) >> 5;
    if (per < 32) per |= 1;
    c.total = total;
    c.off = min(total, (int)(threadIdx.x & 31) * per);
    c.cnt = min(per, total - c.off);
    float s0 = 0.0f, s1 = 0.0f;
    int i = 0;
#pragma unroll 1
    for (; i + 2 <= c.cnt; i += 2) { s0 += list[skew(c.off + i)]; s1 += list[skew(c.off + i + 1)]; }
    if (i < c.cnt) s0 += list[skew(c.off + i)];
    c.csum = s0 + s1;
    return c;
}

__device__ __forceinline__ Item run_item(unsigned int pair, int j, int tile, int cnt, int off, int num) {
    Item it;
    it.ka = pair; it.kb = 0u;
    it.meta = (unsigned int)(j + 127) | (K_RUN << 8) | (255u << 10) | ((unsigned int)tile << 18);
    it.oc = (unsigned int)cnt | ((unsigned int)off << 11) | ((unsigned int)num << 21);
    return it;
}

// The running sum is at least this part of the estimated one: each of the additions before took 2^-24 at most, and the
// estimate does not know that a logit over the temperature and the maximum over it are rounded, by 2^-24 of either.
__device__ __forceinline__ float least_of(int tile, float top) {
    return fmaxf(1.0f - (float)(tile + 1) * ((float)TILE / 16777216.0f) - fabsf(top) * (1.0f / 4194304.0f), 1.0e-6f);
}

// The items of a tile's list cut into chunks, `est` = the estimated sum before the tile. Returns the
// number of items; `care` = this lane's values are wanted one by one.
// `alloc(n, c)` is called by all lanes with the number of items and of careful chunks among them and
// returns where the items go; place(i) says where the i-th careful chunk's values go (255: nowhere).
template <class ALLOC, class PLACE>
__device__ __forceinline__ int tile_items(const float *list, const TileChunk &ch, float est, int tile, float top, ALLOC alloc, PLACE place, bool &care, int &my_place) {
    const int cnt = ch.cnt, off = ch.off, total = ch.total;
    const float csum = ch.csum;
    const int lane = threadIdx.x & 31;
    const float inc = warp_incl_scan(csum, lane);
    float ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = 0.0f;
    const float sst = est + ex;
    const bool nonempty = cnt > 0 && csum > 0.0f;
    // the estimate counts what was dropped (it adds nothing to the true sum), so it is high rather than low
    const float lo = sst * (1.0f - 1.0f / 1024.0f), hi = (sst + csum) * (1.0f + 1.0f / 2048.0f);
    const int jl = fexpo(lo), jh = fexpo(hi);
    const bool usable = nonempty && lo > 0.0f && jh <= jl + 1 && jl >= -100 && jh <= 100;
    const bool two = usable && jh == jl + 1;
    // the lane's values added to the smallest even and the smallest odd pattern of the binade (and of the next):
    // the true sum rounds as the one of its parity does, as long as it stays in the binade
    const unsigned int A1 = (unsigned int)(jl + 127) << 23, A2 = A1 + (1u << 23);
    Units da{0u, 0u}, db{0u, 0u};
    bool bad = false;
    if (__any_sync(0xffffffffu, two)) {
        if (usable) {
            float s0 = __uint_as_float(A1), s1 = __uint_as_float(A1 + 1u), t0 = __uint_as_float(A2), t1 = __uint_as_float(A2 + 1u);
#pragma unroll 2
            for (int i = 0; i < cnt; i++) {
                const float v = list[skew(off + i)];
                s0 = __fadd_rn(s0, v); s1 = __fadd_rn(s1, v);
                t0 = __fadd_rn(t0, v); t1 = __fadd_rn(t1, v);
            }
            da = Units{__float_as_uint(s0) - A1, __float_as_uint(s1) - A1 - 1u};
            db = Units{__float_as_uint(t0) - A2, __float_as_uint(t1) - A2 - 1u};
            bad = __float_as_uint(s1) >= A2 || (two && __float_as_uint(t1) >= A2 + (1u << 23));
        }
    } else if (usable) {
        float s0 = __uint_as_float(A1), s1 = __uint_as_float(A1 + 1u);
#pragma unroll 4
        for (int i = 0; i < cnt; i++) {
            const float v = list[skew(off + i)];
            s0 = __fadd_rn(s0, v); s1 = __fadd_rn(s1, v);
        }
        da = Units{__float_as_uint(s0) - A1, __float_as_uint(s1) - A1 - 1u};
        bad = __float_as_uint(s1) >= A2;
    }
    // A run that adds nothing has no item, unless the sum may still be in the binade below, where it might add something:
    // then it has one of no units, by which the binade is checked.
    const unsigned int um = __ballot_sync(0xffffffffu, usable && (da.even | da.odd) == 0u && fexpo(lo * least_of(tile, top)) < jl);
    const bool step = nonempty && (!usable || bad);
    const unsigned int ne = __ballot_sync(0xffffffffu, nonempty);
    // lanes that round by themselves inside one binade form runs; two neighbours that disagree about
    // the binade do not belong to one run
    const unsigned int below = ne & ((1u << lane) - 1u);
    const int prev = below ? 31 - __clz((int)below) : lane;
    const int pj = __shfl_sync(0xffffffffu, jl, prev);
    const bool prev_alone = ((__ballot_sync(0xffffffffu, step || two) >> prev) & 1u) != 0u;
    care = step || two || (nonempty && below && !prev_alone && pj != jl);
    const unsigned int cm = __ballot_sync(0xffffffffu, care);
    my_place = 255;
    const int j0 = __shfl_sync(0xffffffffu, jl, max(__ffs((int)ne) - 1, 0));
    if (__popc(ne) >= 4 && __all_sync(0xffffffffu, !nonempty || (two && !bad && jl == j0))) {
        // A sum that stays near a power of two for long: most such tiles do not cross it, so several lanes make an item,
        // of 128 values at most, which are in the list. (With an item a lane, one row in some hundreds of 262144 had more
        // careful chunks than row_head takes, and row_tail took 200 us for it.)
        const int lg = total <= 128 ? 5 : (total <= 256 ? 4 : (total <= 512 ? 3 : 2)), in = lane & ((1 << lg) - 1);
        da = units_scan(da, lane, lane - in); db = units_scan(db, lane, lane - in);
        const int first = __shfl_sync(0xffffffffu, off, lane - in), n = 32 >> lg;
        Item *out = alloc(n, 0);
        if (in == (1 << lg) - 1) {
            Item it;
            it.ka = pair_of(da.even, da.odd); it.kb = pair_of(db.even, db.odd);
            it.meta = (unsigned int)(j0 + 127) | (K_DUAL << 8) | (255u << 10) | ((unsigned int)tile << 18);
            it.oc = (unsigned int)(off + cnt - first) | ((unsigned int)first << 11) | ((unsigned int)(lane >> lg) << 21);
            out[lane >> lg] = it;
        }
        return n;
    }
    if (cm == 0u && !__any_sync(0xffffffffu, usable && da.even != da.odd)) {   // one run without a tie
        const unsigned int k = __reduce_add_sync(0xffffffffu, usable ? da.even : 0u);
        if (k == 0u && um == 0u) return 0;
        Item *out = alloc(1, 0);
        if (lane == 0) out[0] = run_item(k, j0, tile, total, 0, 0);
        return 1;
    }
    // the runs between the careful lanes: a run goes with the careful lane behind it, or closes the tile
    const unsigned int lt = (1u << lane) - 1u, cb = cm & lt;
    const int lastc = cb ? 31 - __clz((int)cb) : -1, last = cm ? 31 - __clz((int)cm) : -1;
    const Units k = units_scan(care || !usable ? Units{0u, 0u} : da, lane, care ? lane : lastc + 1);   // of the run up to this lane and with it
    const unsigned int kp = pair_of(k.even, k.odd);
    unsigned int kr = __shfl_up_sync(0xffffffffu, kp, 1);    // of the run that ends before this lane
    if (lane == 0) kr = 0u;
    auto behind = [&](int l) { return l < 0 ? 0xffffffffu : ~((2u << l) - 1u); };   // the lanes past l
    const unsigned int runm = __ballot_sync(0xffffffffu, care && (kr != 0u || (um & lt & behind(lastc)) != 0u));          // careful lanes with a run before them
    const unsigned int ktail = last == 31 ? 0u : __shfl_sync(0xffffffffu, kp, 31);
    const bool tail = ktail != 0u || (um & behind(last)) != 0u;
    const int ncare = __popc(cm), n = ncare + __popc(runm) + (tail ? 1 : 0);
    if (n == 0) return 0;
    Item *out = alloc(n, ncare);
    // the first lane of a run that holds anything, for its binade and its first entry
    auto first_in = [&](int from) { const unsigned int m = ne & ~(from < 0 ? 0u : (from == 31 ? 0xffffffffu : ((2u << from) - 1u))); return m ? __ffs((int)m) - 1 : 31; };
    const int fl = first_in(lastc), tl = first_in(last);
    const int fj = __shfl_sync(0xffffffffu, jl, fl), fo = __shfl_sync(0xffffffffu, off, fl);
    const int tj = __shfl_sync(0xffffffffu, jl, tl), to = __shfl_sync(0xffffffffu, off, tl);
    if (care) {
        int i = __popc(cb) + __popc(runm & lt);
        if ((runm >> lane) & 1u) { out[i] = run_item(kr, fj, tile, off - fo, fo, i); i++; }
        my_place = place(__popc(cb));
        const bool dual = two && !bad;
        Item it;
        it.ka = dual ? pair_of(da.even, da.odd) : 0u;
        it.kb = dual ? pair_of(db.even, db.odd) : 0u;
        it.meta = (dual ? ((unsigned int)(jl + 127) | (K_DUAL << 8)) : (unsigned int)(K_STEP << 8)) | ((unsigned int)my_place << 10) | ((unsigned int)tile << 18);
        it.oc = (unsigned int)cnt | ((unsigned int)off << 11) | ((unsigned int)i << 21);
        out[i] = it;
    }
    if (tail && lane == 0) out[n - 1] = run_item(ktail, tj, tile, total - to, to, n - 1);
    return n;
}

// Most tiles lie inside one binade and hold no tie: their sum is a number of its units, in any order, added up where
// the values are made. (Chunks and items for all tiles took half again as many instructions.) One warp; `est` = the
// estimated sum before the tile, `behind` = the one behind it, as far as it is known: a tile that is expected to leave the binade
// has to be cut into chunks anyway, in short rows nearly every one.
struct QuickSum {
    int j;               // the binade
    bool usable, bad;
    float C, half, big;
    unsigned int k;      // this lane's units; all lanes' once holds() has been true
    __device__ __forceinline__ QuickSum(float est, float behind) {
        const float lo = est * (1.0f - 1.0f / 1024.0f);
        j = fexpo(lo);
        usable = lo > 0.0f && j >= -100 && fexpo(behind * (1.0f + 1.0f / 2048.0f)) == j;
        C = __fmul_rn(1.5f, fpow2(usable ? j : 0)); half = fpow2(usable ? j - 24 : -24); big = fpow2(usable ? j - 1 : -1);
        k = 0u; bad = false;
    }
    __device__ __forceinline__ void add(float e) {
        if (!usable) return;
        const float s = __fadd_rn(e, C);
        k += __float_as_uint(s) - __float_as_uint(C);
        bad |= (fabsf(__fsub_rn(e, __fsub_rn(s, C))) == half) | (e >= big);
    }
    __device__ __forceinline__ bool holds(float est) {
        // (2^23 units, the binade's, or more in a lane: it leaves the binade whatever the others add. Below that 32 lanes do not
        // reach 2^32, which a tile of 1024 values of 2^22 units would: they are no ties and each is below `big`.)
        if (!usable || __any_sync(0xffffffffu, bad || k >= (1u << 23))) return false;
        k = __reduce_add_sync(0xffffffffu, k);
        return fexpo((est + (float)k * fpow2(max(j - 23, -126))) * (1.0f + 1.0f / 2048.0f)) == j;
    }
    // Whether it has an item: see tile_items.
    __device__ __forceinline__ bool counts(float est, int tile, float top) const { return k != 0u || fexpo(est * (1.0f - 1.0f / 1024.0f) * least_of(tile, top)) != j; }
};

struct TileEval { int total; unsigned int keep; };

// The exponentials (temperature and softmax numerator, sample.mojo:419-434) of a tile's logits that
// reach `thr`, packed into the tile's list (over the logits: entry e never lies behind a logit that is
// still to be read). The warp first lists what is kept and then evaluates it in full warps, two of them
// at a time (take(value's bits, second of the two, bit of the time) by the lane that evaluates it); a tile that
// keeps three quarters and more keeps all, and no other has 1024 entries (a value too small to matter adds
// nothing). `idx` holds 1024 positions.
template <class TAKE>
__device__ __forceinline__ TileEval tile_eval(float *tile, unsigned short *idx, float thr, float T, float rT, float top, bool fast, TAKE take) {
    const int lane = threadIdx.x & 31;
    const float *mine = tile + lane * PITCH;
    unsigned int m = 0;
#pragma unroll
    for (int g = 0; g < 8; g++) {
        const float4 v = *reinterpret_cast<const float4 *>(mine + 4 * g);
        m |= (v.x >= thr ? 1u : 0u) << (4 * g) | (v.y >= thr ? 1u : 0u) << (4 * g + 1) | (v.z >= thr ? 1u : 0u) << (4 * g + 2) | (v.w >= thr ? 1u : 0u) << (4 * g + 3);
    }
    TileEval r;
    const int cnt = __popc(m), inc = warp_incl_scan(cnt, lane);
    r.total = __shfl_sync(0xffffffffu, inc, 31);
    const bool all = r.total >= 3 * TILE / 4;
    if (all) { m = 0xffffffffu; r.total = TILE; }
    r.keep = m;
    if (!all) {
        unsigned short *o = idx + (inc - cnt);
        while (m) {
            *o++ = (unsigned short)(lane * 32 + __ffs((int)m) - 1);
            m &= m - 1u;
        }
    }
    __syncwarp();
    const bool one = T == 1.0f;
    auto value = [&](float x) -> float {
        // (what is not there is -inf, which div_by cannot take; everything so far down becomes zero)
        const float v = one ? x : (fast ? div_by(fmaxf(x, -1.0e20f), T, rT) : div_slow(x, T));
        return expf_pinned_nonpos(__fsub_rn(v, top));  // no logit of the row exceeds its maximum
    };
    unsigned int bit = 1u;
#pragma unroll 1
    for (int i0 = 0; i0 < r.total; i0 += 64, bit <<= 1) {
        const int i = i0 + lane, j = i + 32;
        const int p = all ? i : (i < r.total ? (int)idx[i] : 0), q = all ? j : (j < r.total ? (int)idx[j] : 0);
        const float x = tile[p + 4 * (p >> 5)], y = tile[q + 4 * (q >> 5)];
        const float ex = value(x), ey = value(y);
        __syncwarp();
        if (i < r.total) { tile[skew(i)] = ex; take(__float_as_uint(ex), false, bit); }
        if (j < r.total) { tile[skew(j)] = ey; take(__float_as_uint(ey), true, bit); }
        __syncwarp();
    }
    return r;
}

// The careful lanes' values to their places, padded with zeros.
__device__ __forceinline__ void store_care(float *care, const float *list, const TileChunk &ch, int my_place) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (unsigned int left = __ballot_sync(0xffffffffu, my_place != 255); left; left &= left - 1u) {
        const int l = __ffs((int)left) - 1, n = __shfl_sync(0xffffffffu, ch.cnt, l), o = __shfl_sync(0xffffffffu, ch.off, l);
        const int at = __shfl_sync(0xffffffffu, my_place, l);
        care[at * 32 + lane] = lane < n ? list[skew(o + lane)] : 0.0f;
    }
}

// A tile's candidates for the head to their list, or to the second one of F_FAR: `wanted` names, per lane, entries
// entry(b) for every set bit b, with the bits value(e) and the token token(e). A tile asks for its places once. (One
// request per value, each waited for before the next two are evaluated, took 0.7 us each: up to 22 us a tile in short
// rows, whose few tiles hold all candidates.)
template <class ENTRY, class VALUE, class TOKEN>
__device__ __forceinline__ void put_candidates(const RowsArgs &A, int rr, const RowPlan &pl, unsigned int wanted, ENTRY entry, VALUE value, TOKEN token) {
    if (!__any_sync(0xffffffffu, wanted != 0u)) return;
    const int lane = threadIdx.x & 31;
    RowHead *head = A.head(rr);
    auto put = [&](unsigned int m, int *count, unsigned long long *to) {
        const int n = __popc(m), inc = warp_incl_scan(n, lane);
        int pos = 0;
        if (lane == 31 && inc) pos = atomicAdd(count, inc);
        pos = __shfl_sync(0xffffffffu, pos, 31) + inc - n;
#pragma unroll 1
        for (; m; m &= m - 1u, pos++) {
            const int e = entry(__ffs((int)m) - 1);
            if (pos < HEADCAP) to[pos] = make_key(value(e), token(e));
        }
    };
    unsigned int near = wanted;
    if (pl.flags & F_FAR) {
        unsigned int beyond = 0u;
#pragma unroll 1
        for (unsigned int m = wanted; m; m &= m - 1u) {
            const unsigned int eb = value(entry(__ffs((int)m) - 1)), one = m & (0u - m);
            if (eb < pl.tau_bits) near ^= one;
            if (eb >= pl.tau_far && ((pl.flags & F_ALLNEAR) || eb < pl.tau_bits)) beyond |= one;
        }
        put(beyond, &head->nfar, A.far(rr));
    }
    put(near, &head->ncand, A.cand(rr));
}

// The units of binade j that a lane's 32 logits add to a sum there, from hardware exponentials: those whose number
// is certain, added up in `k`; returns which of them are not (and those that reach `tau`, whose value is wanted).
//
// y = ex2(x f + g), f = log2 e / T, g = 23 - j - top log2 e, against Y = expf_pinned(fl(fl(x / T) - top)) 2^(23 - j), of
// which fl adds rne(Y) units. Relative errors in units of 2^-24, for what reaches a quarter of a unit (further down both
// round to nothing), with P = |top| and D = 26 + |j|, the width in powers of two between a quarter of a unit and
// the maximum: f is off by 2, so x f, at most 1.443 P + D, by twice that; g by 1.443 P + D; the sum, of 24 at most where
// it matters, by 24; times ln 2: 3 P + 2.1 D + 17. ex2 by 4. Y itself against exact arithmetic: the quotient by
// P + 0.7 D, the difference by 0.7 D, the exponential by 3. Together 4 P + 3.5 D + 24, and a quarter more here. A y whose
// distance to the nearest integer plus its error stays below a half has the same integer as Y.
constexpr int EXACT_MOST = 256;   // of a tile evaluated in full at most; else all that it keeps is
__device__ __forceinline__ unsigned int near_units(const float *tile, int lane, float T, float top, int j, unsigned int tau, unsigned int &k) {
    const float f = 1.44269504f / T, g = (float)((double)(23 - j) - (double)top * 1.4426950408889634);
    const float err = (5.0f * fabsf(top) + 4.4f * (float)(26 + abs(j)) + 30.0f) * (1.0f / 16777216.0f);
    // (a candidate near the smallest floats is not known by y to within a thousandth: all are evaluated then)
    const float edge = tau < (27u << 23) ? -1.0f : (0.999f - 2.0f * err) * __uint_as_float(tau) * fpow2(min(23 - j, 127)), magic = 12582912.0f;
    const float4 *mine = reinterpret_cast<const float4 *>(tile + lane * PITCH);
    unsigned int m = 0u, sum = 0u;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const float4 v = mine[q];
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float y = ex2_approx(__fmaf_rn(x[u], f, g)), t = __fadd_rn(y, magic), r = __fsub_rn(y, __fsub_rn(t, magic));
            const bool sure = __fmaf_rn(y, err, fabsf(r)) < 0.49999f && y < edge;   // (false for infinities and NaN)
            if (sure) sum += __float_as_uint(t) - __float_as_uint(magic); else m |= 1u << (4 * q + u);
        }
    }
    k = sum;
    return m;
}

__global__ void __launch_bounds__(SPAN_THREADS, 4) tile_exp_kernel(const __grid_constant__ RowsArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SpanShared *S = reinterpret_cast<SpanShared *>(smem_raw);
    pdl_next();
    pdl_wait();
    // (the last spans first: of a block larger than the L2 they are what tile_stats has left there)
    const int b = (int)(gridDim.x - 1u - blockIdx.x), rr = b / A.nspan, span = b - rr * A.nspan, r = A.r0 + rr;
    RowHead *head = A.head(rr);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tile = span * (SPAN / TILE) + warp;
    const size_t gt = (size_t)rr * A.ntile + min(tile, A.ntile - 1);
    const TilePlan tp = A.tp[gt];
    const float tmax = A.ts[gt].tmax;
    if (head->plan.kind == PLAN_DONE) return;
    const bool hot = tile < A.ntile && tmax >= tp.thr;
    const RowPlan pl = head->plan;
    auto store_cold = [&]() {
        if (pl.flags & F_LIST) A.kmask[gt * 32 + lane] = 0u;
        if (lane == 0) { TileOut o; o.ioff = 0u; o.cnt = 0; o.nitem = 0; A.to(rr)[tile] = o; }
    };
    const BatchArgs &a = A.a;
    const RowCfg &c = pl.c;
    // a tile whose maximum does not reach its bound keeps nothing
    if (c.npatch > 0 ? !__syncthreads_or(hot) : !hot) {
        if (tile < A.ntile) store_cold();
        return;
    }
    if (hot) span_fetch(a, c.lrow, span * SPAN, S->x);
    span_ready(a, c, r, span * SPAN, S->x, &S->s, true, hot);
    if (tile >= A.ntile) return;
    if (!hot) { store_cold(); return; }
    float *list = S->x + (size_t)warp * 32 * PITCH;
    const unsigned int tau = min(pl.tau_bits, pl.tau_far);
    unsigned short *idx = reinterpret_cast<unsigned short *>(S->s.cnt) + warp * TILE;
    QuickSum qs(tp.est, tile + 1 < A.ntile ? A.tp[gt + 1].est : tp.est);
    auto add_units = [&](float e) { qs.add(e); };
    int ni = 0, cnt = TILE;
    unsigned int i0 = 0u;
    auto store_out = [&]() {
        if (lane != 0) return;
        TileOut o;
        o.ioff = i0; o.cnt = (unsigned short)cnt; o.nitem = (unsigned short)ni;
        A.to(rr)[tile] = o;
    };
    auto store_run = [&]() {
        ni = qs.counts(tp.est, tile, pl.top) ? 1 : 0;
        if (lane == 0 && ni) {
            i0 = (unsigned int)atomicAdd(&head->nitem, 1);
            A.items(rr)[i0] = run_item(qs.k, qs.j, tile, cnt, 0, 0);
        }
    };
    const bool fast = (pl.flags & F_FASTDIV) && tp.thr > -INFINITY;
    const float rT = __fdiv_rn(1.0f, c.T);
    if (qs.usable && fast && !(pl.flags & F_LIST)) {
        // Nobody asks for this row's list, only for its sum and its candidates, and nearly all that is kept adds
        // few units, whose number a hardware exponential tells unless it is near a half: see near_units. The others
        // are evaluated as they have to be. Per tile 600 instructions, where evaluating all that is kept takes 1300
        // (at a fifth of the logits kept: 1024 rows of 262144 with a top-k of 1024, 450 us).
        const unsigned int m = near_units(list, lane, c.T, pl.top, qs.j, tau, qs.k);
        const int mine = __popc(m), inc = warp_incl_scan(mine, lane), total = __shfl_sync(0xffffffffu, inc, 31);
        if (total <= EXACT_MOST) {
            float *val = reinterpret_cast<float *>(idx + EXACT_MOST);
            unsigned short *o = idx + (inc - mine);
#pragma unroll 1
            for (unsigned int w = m; w; w &= w - 1u) *o++ = (unsigned short)(lane * 32 + __ffs((int)w) - 1);
            __syncwarp();
            unsigned int wanted = 0u, bit = 1u;
            const bool one = c.T == 1.0f;
#pragma unroll 1
            for (int i = lane; i - lane < total; i += 32, bit <<= 1) {
                const int p = i < total ? (int)idx[i] : 0;
                const float x = list[p + 4 * (p >> 5)];
                if (i < total && x >= tp.thr) {   // (not a number: never kept)
                    const float e = expf_pinned_nonpos(__fsub_rn(one ? x : div_by(x, c.T, rT), pl.top));
                    add_units(e);
                    val[i] = e;
                    if (__float_as_uint(e) >= tau) wanted |= bit;
                }
            }
            __syncwarp();
            if (qs.holds(tp.est)) {
                put_candidates(A, rr, pl, wanted, [&](int b) { return b * 32 + lane; }, [&](int e) { return __float_as_uint(val[e]); },
                               [&](int e) { return tile * TILE + (int)idx[e]; });
                store_run();
                store_out();
                return;
            }
            __syncwarp();
        }
        qs.k = 0u; qs.bad = false;
    }
    unsigned int w0 = 0u, w1 = 0u;   // this lane's candidates among the entries it evaluates
    const TileEval t = tile_eval(list, idx, tp.thr, c.T, rT, pl.top, fast,
        [&](unsigned int eb, bool second, unsigned int bit) {
            if (eb >= tau) { if (second) w1 |= bit; else w0 |= bit; }
            add_units(__uint_as_float(eb));
        });
    cnt = t.total;
    put_candidates(A, rr, pl, w0 | (w1 << 16), [&](int b) { return (b & 15) * 64 + (b & 16) * 2 + lane; },
                   [&](int e) { return __float_as_uint(list[skew(e)]); }, [&](int e) { return tile * TILE + (t.total == TILE ? e : (int)idx[e]); });
    bool whole = (pl.flags & F_LIST) != 0;
    if (qs.holds(tp.est)) store_run();
    else {
        const TileChunk ch = tile_chunk(list, t.total);
        bool care;
        int my_place, c0 = CARE_PLACES;
        ni = tile_items(list, ch, tp.est, tile, pl.top,
            [&](int n, int nc) -> Item * {
                if (lane == 0) { i0 = (unsigned int)atomicAdd(&head->nitem, n); if (nc) c0 = atomicAdd(&head->ncare, nc); }
                i0 = __shfl_sync(0xffffffffu, i0, 0); c0 = __shfl_sync(0xffffffffu, c0, 0);
                return A.items(rr) + i0;
            },
            [&](int i) { return c0 + i < CARE_PLACES ? c0 + i : 255; }, care, my_place);
        store_care(A.care(rr), list, ch, my_place);
        whole = whole || __any_sync(0xffffffffu, care && my_place == 255);
    }
    if (whole)
#pragma unroll 1
        for (int i = lane; i < t.total; i += 32) A.elist[gt * TILE + i] = list[skew(i)];
    if (pl.flags & F_LIST) A.kmask[gt * 32 + lane] = t.keep;
    store_out();
}

// =============================================================================
// Kernel 4: one small block per sampled row. The items give the softmax denominator, the candidates the
// sorted head; most rows end here. Rows that go on (nothing sorted, a nucleus past the head, typical-p,
// anything unusual) are queued for the last kernel. Bound: the latency of one warp's dependent additions
// and of one round of loads, so the block is small and four of them share an SM: 20 us for
// 64 rows, 34 for 256, 42 for 512 with a top-k of 1024 (three an SM, two rounds of them: 60). (Run by the tail's 512 threads, one block an SM, the same
// rows took twice as long.)
// =============================================================================
constexpr int HT = 256, HW = HT / 32;
constexpr int H_ITEMS = 1024;              // items of a row
constexpr int H_CARE = 64, H_REC = 704;    // careful chunks whose values are at hand, and all of them (what four blocks an SM have room for)
// What a queued row has: nothing; its denominator; its head too (tile_walk prepares the walk past it);
// its denominator, and nothing to be sorted (tile_walk prepares the sum of the probabilities).
enum { ST_NOTHING = 0, ST_SUM = 1, ST_HEAD = 2, ST_PURE = 3, ST_DONE = 4 };

struct __align__(16) CareRec { unsigned int k, meta, ka, kb; };   // units of all runs before it; binade of the one right before it, or 0 | kind | own binade | place

struct __align__(16) WalkShared {
    Item items[H_ITEMS];
    float care[H_CARE * 32];
    union {
        unsigned short toff[MAX_TILES + 4];   // the tiles' first items, until these are in order
        CareRec rec[H_REC + 1];
    };
    unsigned int sbs[H_REC + 2];           // the sum before every record's runs
    unsigned short ritem[H_REC];
    unsigned int ws[NWARP + 1], ws2[NWARP + 1];
};

struct __align__(16) HeadShared {
    union {
        WalkShared w;
        struct {   // once the sum is known
            union {
                unsigned int sbin[NBINS];
                struct { unsigned long long keys[HEADC]; float lg[HEADC], tt[HEADC]; } typ;
            };
            union {
                unsigned long long tmp[HEADCAP];
                struct { float pc[HEADCAP]; float pre[HEADCAP]; } p;
            };
        };
    };
    unsigned long long cand[HEADCAP];
    unsigned int ws[HW + 1], ws2[HW + 1];
    float Z; int ok, cut, n_ge; unsigned int tie;
    float ent;
};
static_assert(4 * (sizeof(HeadShared) + 1024) <= 228 * 1024, "four blocks an SM");

// Everything about a row's items, in one round of loads by N threads (what lies past the counts is not used).
template <int N>
struct WalkLoads {
    static constexpr int TPT = (MAX_TILES + N - 1) / N, IPT = (H_ITEMS + N - 1) / N, CV = (H_CARE * 8 + N - 1) / N;
    TileOut to[TPT];
    Item it[IPT];
    float4 cv[CV];
    __device__ __forceinline__ void load(const RowsArgs &R, int rr) {
        const int tid = threadIdx.x;
#pragma unroll
        for (int u = 0; u < TPT; u++) {
            to[u].nitem = 0;
            if (TPT * tid + u < R.ntile) to[u] = R.to(rr)[TPT * tid + u];
        }
#pragma unroll
        for (int u = 0; u < IPT; u++)
            if (tid + u * N < H_ITEMS) it[u] = R.items(rr)[tid + u * N];
#pragma unroll
        for (int u = 0; u < CV; u++)
            if (tid + u * N < H_CARE * 8) cv[u] = reinterpret_cast<const float4 *>(R.care(rr))[tid + u * N];
    }
    // The items in order, the careful ones among them as records; returns the number of records.
    __device__ __forceinline__ unsigned int order(WalkShared *W, int ntile, int nitem) {
        const int tid = threadIdx.x;
        unsigned int total, n0 = 0u;
#pragma unroll
        for (int u = 0; u < TPT; u++) n0 += to[u].nitem;
        unsigned int o = head_scan<N>(n0, W->ws, &total);
#pragma unroll
        for (int u = 0; u < TPT; u++) {
            if (TPT * tid + u < ntile) W->toff[TPT * tid + u] = (unsigned short)o;
            o += to[u].nitem;
        }
#pragma unroll
        for (int u = 0; u < CV; u++)
            if (tid + u * N < H_CARE * 8) reinterpret_cast<float4 *>(W->care)[tid + u * N] = cv[u];
        __syncthreads();
#pragma unroll
        for (int u = 0; u < IPT; u++)
            if (tid + u * N < nitem) W->items[W->toff[it[u].tile()] + it[u].num()] = it[u];
        __syncthreads();
        unsigned int pj[IPT], k = 0u, n = 0u, care = 0u;
#pragma unroll
        for (int u = 0; u < IPT; u++) {
            const int i = IPT * tid + u;
            pj[u] = 0u;
            if (i < nitem) {
                it[u] = W->items[i];
                const bool run = it[u].kind() == K_RUN;
                bool prev_run = false;
                if (i > 0) { const Item p = W->items[i - 1]; prev_run = p.kind() == K_RUN; pj[u] = prev_run ? p.jb() : 0u; }
                if (!run || !parity_free(it[u].ka) || (prev_run && pj[u] != it[u].jb())) { care |= 1u << u; n++; }   // (a change of binade between two runs: a wrong guess)
                else k += it[u].ka;
            }
        }
        unsigned int ktot, nrec;
        unsigned int kx = head_scan<N>(k, W->ws, &ktot), nx = head_scan<N>(n, W->ws2, &nrec);
        if (nrec <= (unsigned int)H_REC) {
#pragma unroll
            for (int u = 0; u < IPT; u++) {
                const int i = IPT * tid + u;
                if (i >= nitem) break;
                if ((care >> u) & 1u) {
                    CareRec c;
                    c.k = kx; c.ka = it[u].ka; c.kb = it[u].kb;
                    c.meta = pj[u] | (it[u].kind() << 8) | (it[u].jb() << 16) | (it[u].place() << 24);
                    W->ritem[nx] = (unsigned short)i;
                    W->rec[nx++] = c;
                } else kx += it[u].ka;
            }
            if (tid == 0) {
                CareRec c;
                c.k = ktot; c.ka = c.kb = 0u; c.meta = nitem > 0 && W->items[nitem - 1].kind() == K_RUN ? W->items[nitem - 1].jb() : 0u;
                W->rec[nrec] = c;
            }
        }
        __syncthreads();
        return nrec;
    }
};

// One warp, all lanes alike: the sum through the careful chunks W->rec[0..nrec) and the runs between
// them; `more` holds the values of all of them. Returns false where a run's binade was guessed wrong.
// Bound: 32 dependent additions a careful chunk, and the fetch of instructions: one warp runs this, once.
// A register that has been added takes the next record's value at once, so that no load is waited for
// between two chunks (337 cycles a record when each asked for its own; two sets of registers spill).
// Chunks whose sum may lie in either of two binades come in stretches wherever a row's sum stays near a
// power of two for long, 188 in one row of 196: while the binade holds, 32 of them are one prefix sum over
// the lanes (173 cycles each one after the other), out of line, because most rows have none. Only behind four in a row:
// most come by twos and threes before a crossing, and the prefix sum, tried there, took nothing and 700 cycles (100 rows
// of 50257 9.3 thousand cycles where they now take 7.7, the longest 18.8 and 14.6).
__device__ __forceinline__ unsigned int kind_of(const CareRec &c) { return (c.meta >> 8) & 3u; }
// From record q on: how many records one prefix sum takes, and the sum behind them.
__device__ __noinline__ uint2 dual_stretch(WalkShared *W, int nrec, int q, unsigned int sb, unsigned int kdone) {
    const int lane = threadIdx.x & 31;
    const unsigned int e = sb >> 23;
    CareRec c;
    c.k = 0u; c.meta = 0u; c.ka = c.kb = 0u;
    if (q + lane < nrec) c = W->rec[q + lane];
    unsigned int kp = __shfl_up_sync(0xffffffffu, c.k, 1);
    if (lane == 0) kp = kdone;
    const unsigned int runs = c.k - kp, jb = (c.meta >> 16) & 0xffu, kind = kind_of(c), own = e == jb ? c.ka : c.kb;
    const bool can = q + lane < nrec && (kind == K_DUAL ? (e == jb || e == jb + 1u) : (kind == K_RUN && e == jb && (own & 0x3fffffffu) < (1u << 24))) &&
                     ((c.meta & 0xffu) == 0u || ((c.meta & 0xffu) == e && runs < (1u << 24)));
    Units d{0u, 0u};
    if (can) d = Units{runs + units(own, runs), runs + units(own, runs + 1u)};
    d = units_scan(d, lane, 0);
    const unsigned int inc = (sb & 1u) ? d.odd : d.even;
    const unsigned int stop = __ballot_sync(0xffffffffu, !can || ((sb + inc) >> 23) != e);
    const int n = stop ? __ffs((int)stop) - 1 : 32;
    unsigned int before = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) before = 0u;
    if (lane < n) W->sbs[q + lane] = sb + before;
    if (n > 0) sb += __shfl_sync(0xffffffffu, inc, n - 1);
    return make_uint2(sb, (unsigned int)n);
}
__device__ __noinline__ float add_listed(float s, const float *v, int n) {
    const int lane = threadIdx.x & 31;
    float next = lane < n ? v[lane] : 0.0f;
#pragma unroll 1
    for (int i = 0; i < n; i += 32) {
        const float mine = next;
        next = i + 32 + lane < n ? v[i + 32 + lane] : 0.0f;
#pragma unroll 8
        for (int e = 0; e < 32; e++) s = __fadd_rn(s, __shfl_sync(0xffffffffu, mine, e));
    }
    return s;
}
__device__ __forceinline__ bool walk_records(WalkShared *W, const float *more, const float *list, int nrec, float &Z) {
    unsigned int sb = 0u, kdone = 0u;
    CareRec r = W->rec[0], nx = W->rec[min(1, nrec)];
    auto values = [&](const CareRec &c) { return reinterpret_cast<const float4 *>(W->care + min(c.meta >> 24, (unsigned int)H_CARE - 1u) * 32); };
    float4 x[8];
    {
        const float4 *v = values(r);
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = v[i];
    }
    bool fine = true;
    int inside = 0;   // records in a row that needed no additions
#pragma unroll 1
    for (int q = 0; ; q++) {
        const float4 *v = values(nx);   // the next record's
        const CareRec c = r;
        r = nx;
        nx = W->rec[min(q + 2, nrec)];
        W->sbs[q] = sb;
        const unsigned int to = sb + (c.k - kdone), j = c.meta & 0xffu, kind = kind_of(c), jb = (c.meta >> 16) & 0xffu, place = c.meta >> 24;
        if (j != 0u && ((sb >> 23) != j || (to >> 23) != j)) { fine = false; break; }   // (also where the runs add nothing)
        kdone = c.k;
        sb = to;
        if (q == nrec) break;
        const bool run = kind == K_RUN, low = (sb >> 23) == jb;
        const unsigned int e = sb >> 23, td = sb + units(low ? c.ka : c.kb, sb);
        if (run && (!low || (td >> 23) != jb)) { fine = false; break; }
        if (run || (kind == K_DUAL && (low || e == jb + 1u) && (td >> 23) == e)) {
            sb = td;
            if (++inside >= 4 && q + 6 < nrec && kind_of(r) != K_STEP && kind_of(nx) != K_STEP && kind_of(W->rec[q + 6]) != K_STEP) {
                const uint2 t = dual_stretch(W, nrec, q + 1, sb, kdone);
                sb = t.x;
                q += (int)t.y;
                kdone = t.y ? W->rec[q].k : kdone;
                if (t.y < 8u) inside = 0;
                r = W->rec[q + 1];
                nx = W->rec[min(q + 2, nrec)];
                v = values(r);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = v[i];
            continue;
        }
        inside = 0;
        if (place >= H_CARE) {   // (a row with many: their values are still in L2)
            if (place == 255u) {   // (past CARE_PLACES, or several lanes' values: in its tile's list)
                const Item it = W->items[W->ritem[q]];
                sb = __float_as_uint(add_listed(__uint_as_float(sb), list + (size_t)it.tile() * TILE + it.off(), it.cnt()));
#pragma unroll
                for (int i = 0; i < 8; i++) x[i] = v[i];
                continue;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = reinterpret_cast<const float4 *>(more + place * 32)[i];
        }
        float s = __uint_as_float(sb);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, x[i].x), x[i].y), x[i].z), x[i].w);
            x[i] = v[i];
        }
        sb = __float_as_uint(s);
    }
    W->sbs[nrec + 1] = sb;
    Z = __uint_as_float(sb);
    return fine;
}

// Typical-p (sample.mojo:525-567) on the m kept probabilities S->p.pc[0..m), descending, ids in S->cand:
// entropy H = -sum p log p added up in that order, distance |-log p - H|, stable order by distance, the
// smallest prefix whose probabilities add up to typ, the draw (:569-594) over that prefix in that order.
__device__ __noinline__ void typical_rows(HeadShared *S, const BatchArgs &a, int r, const RowCfg &g, int m, float Z, unsigned int status) {
    const int tid = threadIdx.x;
    const float *pc = S->p.pc;
    float *pre = S->p.pre;
    unsigned long long *keys = S->typ.keys;
    if (m <= 0 || m > HEADC) {   // what the earlier filters left reaches past the head, or is wider than the filter's scratch
        if (tid == 0) finish_row(a, r, g, status | MOLLA_ROW_UNSUPPORTED, -1, Z, 0, 0, 0);
        return;
    }
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < m; i += HT) {
        const float p = pc[i];
        const float l = (p > 0.0f) ? logf_pinned(p) : 0.0f;
        S->typ.lg[i] = l;
        S->typ.tt[i] = (p > 0.0f) ? __fmul_rn(p, l) : 0.0f;
    }
    __syncthreads();
    if (tid == 0) {
        float ent = 0.0f;
#pragma unroll 1
        for (int i = 0; i < m; i++)
            if (pc[i] > 0.0f) ent = __fsub_rn(ent, S->typ.tt[i]);
        S->ent = ent;
    }
    __syncthreads();
    const float ent = S->ent;
    constexpr int KPT = HEADC / HT;
    unsigned long long k[KPT];
    int rank[KPT];
#pragma unroll
    for (int u = 0; u < KPT; u++) {
        const int i = tid + u * HT;
        k[u] = 0ull; rank[u] = 0;
        if (i < m) {
            const float sur = (pc[i] > 0.0f) ? -S->typ.lg[i] : 0.0f;
            const float d = fabsf(__fsub_rn(sur, ent));
            // descending keys = ascending distance, and among equal distances ascending position (stable)
            k[u] = ((unsigned long long)(~__float_as_uint(d)) << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned int)i);
            keys[i] = k[u];
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int j = 0; j < m; j++) {
        const unsigned long long o = keys[j];
#pragma unroll
        for (int u = 0; u < KPT; u++) rank[u] += o > k[u] ? 1 : 0;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < KPT; u++)
        if (tid + u * HT < m) keys[rank[u]] = k[u];
    __syncthreads();
    if (tid == 0) {
        auto at_of = [&](int j) { return (int)(0xFFFFFFFFu - (unsigned int)(keys[j] & 0xFFFFFFFFull)); };
        float s = 0.0f;
        int kept = m;
#pragma unroll 1
        for (int j = 0; j < m; j++) {
            s = __fadd_rn(s, pc[at_of(j)]);
            pre[j] = s;
            if (s >= g.typ) { kept = j + 1; break; }
        }
        const float sum = pre[kept - 1];
        int at = kept - 1;
        float target = 0.0f;
        if (sum <= 0.0f) at = 0;  // sample.mojo:583-584
        else {
            target = __fmul_rn(draw01(a.seed ? a.seed[g.q] : 0ull, a.drawn ? a.drawn[g.q] : 0ull), sum);
#pragma unroll 1
            for (int j = 0; j < kept; j++)
                if (target < pre[j]) { at = j; break; }
        }
        const int i = at_of(at);
        if ((i > 0 && pc[i - 1] == pc[i]) || (i + 1 < HEADCAP && pc[i + 1] == pc[i])) status |= MOLLA_ROW_CHOSEN_TIE;
        // the last one kept and the first one dropped equally probable: which of them the reference
        // keeps depends on the order its sort left them in
        if (kept < m && pc[at_of(kept - 1)] == pc[at_of(kept)]) status |= MOLLA_ROW_TOPP_TIE;
        finish_row(a, r, g, status, key_idx(S->cand[i]), Z, sum, target, pc[i]);
    }
}

// (PER_SM blocks an SM: with four its registers spill, which 300 rows of 8000 with a top-k pay for, 54 us where three take 52)
template <int PER_SM>
__global__ void __launch_bounds__(HT, PER_SM) row_head_kernel(const __grid_constant__ RowsArgs R) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HeadShared *S = reinterpret_cast<HeadShared *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rr = blockIdx.x, r = R.r0 + rr;
    pdl_next();
    pdl_wait();
    RowHead *head = R.head(rr);
    const BatchArgs &a = R.a;
    const int ntile = R.ntile;
    // everything that will be wanted, in one round of loads (what lies past the counts is not used)
    const int ncand = head->ncand, nitem = head->nitem;
    const RowPlan &pl = head->plan;
    const int kind = pl.kind;
    WalkLoads<HT> wl;
    wl.load(R, rr);
    unsigned long long key = R.cand(rr)[tid];
    if (kind == PLAN_DONE) return;
    const RowCfg &g = pl.c;
    const bool all_near = (pl.flags & F_ALLNEAR) != 0;
    const int nfar = (pl.flags & F_FAR) ? head->nfar : 0, nfirst = all_near ? 0 : ncand;   // of the near list, with the far one
    const bool far = nfar > 0 && nfirst + nfar <= HEADCAP && (!all_near || (ncand > HEADCAP && (g.open_row || nfar >= pl.need)));
    const int nc = far ? nfirst + nfar : ncand;
    // (the near head alone, or what the general form makes of it, would have walked on from here)
    const int nwalk = far && g.n_lim + 1 > (g.open_row ? HEAD_NEED : HEAD_MOST) ? (all_near ? pl.need : ncand) : nc;
    const bool narrow = (pl.flags & F_NARROW) != 0;
    auto queue_row = [&](int state, int why = 0) {
#ifdef MOLLA_SAMPLE_TESTING
        if (a.prof && tid == 0) { a.prof[(long long)r * 32 + 24] = why; a.prof[(long long)r * 32 + 25] = nitem; a.prof[(long long)r * 32 + 26] = head->ncare; a.prof[(long long)r * 32 + 27] = ncand; }
#endif
        if (tid == 0) { head->state = state; R.queue[1 + atomicAdd(&R.queue[0], 1)] = rr; }
    };
    if (nitem > H_ITEMS || (!g.pure && nc > HEADCAP)) { queue_row(ST_NOTHING, 1); return; }
    const unsigned long long seed = a.seed ? a.seed[g.q] : 0ull, drawn = a.drawn ? a.drawn[g.q] : 0ull;   // (not needed before the end)
    if (tid == 0) S->n_ge = 0;
    const unsigned int nrec = wl.order(&S->w, ntile, nitem);
    if (nrec > (unsigned int)H_REC) { queue_row(ST_NOTHING, 2); return; }
    // ---- the softmax denominator, exactly as the sequential loop rounds it (sample.mojo:431-434)
    if (warp == 0) {
        float z = 0.0f;
        const bool fine = walk_records(&S->w, R.care(rr), R.elist + (size_t)rr * ntile * TILE, (int)nrec, z);
        if (lane == 0) { S->Z = z; S->ok = fine ? 1 : 0; }
    }
    __syncthreads();
    if (!S->ok) { queue_row(ST_NOTHING, 3); return; }
    const float Z = S->Z, yZ = __fdiv_rn(1.0f, Z);
    if (tid == 0) head->Z = Z;
    if (g.pure) {
        if (g.minp > 0.0f) { queue_row(ST_SUM, 4); return; }   // (what min-p leaves out is in no estimate)
        if (tid == 0) { head->nitem = 0; head->ncare = 0; }
        queue_row(ST_PURE, 4);
        return;
    }
    // ---- sorted order: the head's candidates as probabilities
#pragma unroll 1
    for (int i = tid; i < nc; i += HT) {
        if (far && i >= nfirst) key = R.far(rr)[i - nfirst];
        else if (i >= HT) key = R.cand(rr)[i];
        S->cand[i] = ((unsigned long long)__float_as_uint(prob_of(key_val(key), Z, yZ)) << 32) | (key & 0xFFFFFFFFull);
    }
    __syncthreads();
    sort_keys<HT, HT>(nc, S->cand, S->tmp, S->p.pc, S->sbin, S->ws, S->ws2);
    // min-p (sample.mojo:508-523) keeps a prefix of the sorted order: what reaches p_max * min_p
    long long n_use = g.n_lim;
    bool all_above = false;   // every candidate does: how many others do is not known here
    if (g.minp > 0.0f) {
        const float floor_p = __fmul_rn(__fdiv_rn(expf_pinned(__fsub_rn(pl.top, pl.top)), Z), g.minp);
        if (!(floor_p >= 2.2e-8f)) {
            if (tid == 0) finish_row(a, r, g, MOLLA_ROW_UNSUPPORTED | (narrow ? MOLLA_ROW_SLOW_PATH : 0u), -1, Z, 0, 0, 0);
            if (pl.flags & F_JUMP) queue_row(ST_DONE, 7);
            return;
        }
        int n = 0;
#pragma unroll 1
        for (int i = tid; i < nc; i += HT) n += S->p.pc[i] >= floor_p ? 1 : 0;
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0 && n) atomicAdd(&S->n_ge, n);
        __syncthreads();
        const int n_ge = max(1, S->n_ge);
        all_above = S->n_ge == nc;
        if (!all_above && n_ge < n_use) n_use = n_ge;
    }
#ifdef MOLLA_SAMPLE_TESTING
    if (a.topk_out) {
#pragma unroll 1
        for (int i = tid; i < a.topk_cap; i += HT)
            a.topk_out[(long long)r * a.topk_cap + i] = (i < nc && (long long)i < n_use) ? key_idx(S->cand[i]) : -1;
    }
#endif
    if (warp == 0) {
        const HeadEnd e = head_end(HeadRule{g.n_lim, g.P, g.open_row, g.topp_on, g.typ < 1.0f}, a.V, S->p.pc, S->p.pre, nc, nwalk, n_use, narrow, false, draw01(seed, drawn));
        if (lane == 0) {
            if (e.at >= 0)
                finish_row(a, r, g, e.tie | (narrow ? MOLLA_ROW_SLOW_PATH : 0u), key_idx(S->cand[e.at]), Z, e.sum, e.target, S->p.pc[e.at]);
            else if (!(g.typ < 1.0f)) {
                head->head_s = e.s; head->head_pos = e.pos;
            }
            S->cut = e.cut; S->tie = e.tie;
        }
    }
    __syncthreads();
    if (g.typ < 1.0f) {
        typical_rows(S, a, r, g, narrow ? -1 : S->cut, Z, S->tie | (narrow ? MOLLA_ROW_SLOW_PATH : 0u));
        if (pl.flags & F_JUMP) queue_row(ST_DONE, 7);
        return;
    }
    if (S->cut > 0) {
        if (pl.flags & F_JUMP) queue_row(ST_DONE, 7);
        return;
    }
    if (all_above || nc == 0) { queue_row(ST_SUM, 5); return; }
    // past the head: the sorted candidates and their prefix sums go along, and empty tables for tile_walk
    {
        ulonglong2 *z = reinterpret_cast<ulonglong2 *>(R.table(rr, 0));
#pragma unroll 1
        for (int i = tid; i < WALK_BINADES * NBINS / 2; i += HT) z[i] = make_ulonglong2(0ull, 0ull);
        if (tid < WALK_BINADES) R.ties(rr)[tid].n = 0;
        if (tid == 0) { R.picks(rr)->n = 0; R.picks(rr)->arrived = 0; }
    }
#pragma unroll 1
    for (int i = tid; i < nc; i += HT) { R.cand(rr)[i] = S->cand[i]; R.pre(rr)[i] = S->p.pre[i]; }
    if (far && tid == 0) { head->ncand = nc; head->plan.tau_bits = pl.tau_far; }
    queue_row(ST_HEAD, 6);
}

// =============================================================================
// Kernel 5: the lists of queued rows, a tile per warp: exponentials become probabilities p = e / Z
// (sample.mojo:437-438). Where nothing is sorted, the items of their sum in vocabulary order; past a
// sorted head, the bin tables of the walk in the binades the sum will go through: an element adds
// rne(p / ulp) units to whatever sum lies in the binade, so one histogram of those integers per binade
// tells where the sum crosses anything. Blocks take spans from the queue as long as there are any.
// Bound: the latency of dependent instructions, branches and loads; 37 us for 58
// rows of 151936 past the head (with every element added to all three tables, and every block's tables to the row's: 48), 14 for 48 rows of 50257 that sort nothing. In the row's own block the same passes took 100 us and more.
// =============================================================================
union __align__(16) WalkTileShared {
    float x[SPAN_THREADS * PITCH];
    struct {
        unsigned int hq[WALK_BINADES][NBINS];   // the low MASS_SPLIT bits of the contributions, summed, and the rest
        unsigned int hqh[WALK_BINADES][NBINS];
    };
};

struct PlanFind { double ws[SPAN_THREADS / 32]; double before, end, total; int hit; unsigned int prev; int next; int pick[PICKS], n; };

// In a walk's table `tab` below bin `hi`, with m0 units before it: the first bin from the top whose end
// reaches x units (F.hit, or -1), the units before and behind it, its neighbours that hold anything, and
// the units of all bins.
__device__ __noinline__ void plan_find(PlanFind &F, const unsigned long long *tab, int hi, double m0, double x) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = NBINS / SPAN_THREADS;
    const int top = NBINS - 1 - PER * tid;
    unsigned long long q[PER], sum = 0ull;
#pragma unroll
    for (int i = 0; i < PER; i++) { q[i] = top - i < hi ? __ldcg(tab + top - i) : 0ull; sum += q[i]; }
    const double inc = warp_incl_scan((double)sum, lane);
    __syncthreads();
    if (lane == 31) F.ws[warp] = inc;
    if (tid == 0) { F.hit = -1; F.prev = 0xffffffffu; F.next = -1; }
    __syncthreads();
    double b0 = 0.0, t = 0.0;
#pragma unroll 1
    for (int w = 0; w < SPAN_THREADS / 32; w++) { if (w == warp) b0 = t; t += F.ws[w]; }
    if (tid == 0) F.total = t;
    double c = m0 + b0 + (inc - (double)sum);
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int b = top - i;
        const double v = (double)q[i];
        if (v > 0.0) {
            if (c < x && c + v >= x) { F.hit = b; F.before = c; F.end = c + v; }
            if (c + v < x) atomicMin(&F.prev, (unsigned int)b);   // the last one before it
            if (c >= x) atomicMax(&F.next, b);                    // the first one behind it
        }
        c += v;
    }
    __syncthreads();
}
__device__ __forceinline__ void plan_want(PlanFind &F, int b) {   // one thread
    if (b < 0 || b >= NBINS) return;
#pragma unroll 1
    for (int i = 0; i < F.n; i++) if (F.pick[i] == b) return;
    if (F.n < PICKS) F.pick[F.n++] = b;
}

// Which bins the walk past row rr's head will look into element by element: from the tables alone the
// sum before every bin is known to within the rounding inside one bin and a few ties, so the bins where it
// crosses into the next binade, reaches top-p, or passes the drawn target are known but for a neighbour.
// What is left out here is only slower: row_tail then looks for it in the list.
__device__ __noinline__ void plan_picks(const RowsArgs &R, int rr, float hs, int j0, int nb) {
    __shared__ PlanFind F;
    const int tid = threadIdx.x, lane = tid & 31;
    const RowCfg &g = R.head(rr)->plan.c;
    double start[WALK_BINADES];
    int hi_of[WALK_BINADES], low_of[WALK_BINADES];
    double s = (double)hs, sum_lo = s, sum_hi = s, unsure = 0.0;   // unsure: how far s may be off
    int hi = NBINS, phases = 0;
    if (tid == 0) F.n = 0;
    // stretch p: the running sum in binade j0 + p
#pragma unroll
    for (int p = 0; p < WALK_BINADES; p++) {
        start[p] = s; hi_of[p] = hi; low_of[p] = 0;
        if (p >= nb || hi <= 0) continue;
        const double unit = dpow2(j0 + p - 23), inv = dpow2(23 - j0 - p);
        double x = 16777216.0;
        const double cut = g.topp_on ? ceil((double)g.P * inv) : 1.0e30;
        const bool by_cut = cut <= x;
        if (by_cut) x = cut;
        plan_find(F, R.table(rr, p), hi, s * inv, x);
        phases = p + 1;
        const int hb = F.hit;
        if (hb < 0) { s = s + F.total * unit; sum_lo = sum_hi = s; hi = 0; continue; }
        low_of[p] = hb;
        // the ties down to that bin add to the sum but are not in the table
        const WalkTies *t = R.ties(rr) + p;
        const int nt = min(__ldcg(&t->n), TIE_CAP);
        float tied = 0.0f;
#pragma unroll 1
        for (int i = lane; i < nt; i += 32) {
            const unsigned int b = (unsigned int)(__ldcg(&t->key[i]) >> 32);
            if ((int)(b >> BIN_SHIFT) >= hb && (int)(b >> BIN_SHIFT) < hi) tied += __uint_as_float(b);
        }
        const double more = (double)warp_sum(tied) * inv, slack = 96.0 + unsure * inv;
        if (tid == 0) {
            plan_want(F, hb);
            if (x - F.before < slack + more) plan_want(F, (int)F.prev);
            if (F.end - x < slack) plan_want(F, F.next);
        }
        s = F.end * unit + more * unit;
        // the elements of that bin behind the crossing add units of the next binade
        if (!by_cut && p + 1 < nb) unsure += fabs((double)__ldcg(R.table(rr, p) + hb) * unit - (double)__ldcg(R.table(rr, p + 1) + hb) * 2.0 * unit);
        sum_lo = sum_hi = s;
        if (by_cut) { sum_lo = x * unit; sum_hi = fmin(s, (x + slack) * unit + (double)__uint_as_float((unsigned int)(hb + 1) << BIN_SHIFT)); }
        hi = by_cut ? 0 : hb;
        __syncthreads();
    }
    // the draw
    const BatchArgs &a = R.a;
    const double u01 = (double)draw01(a.seed ? a.seed[g.q] : 0ull, a.drawn ? a.drawn[g.q] : 0ull);
    int last = -1;
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const double tg = k == 0 ? u01 * sum_lo * (1.0 - 1.0e-6) : u01 * sum_hi * (1.0 + 1.0e-6);
        if (tg < (double)hs) continue;   // in the head
        int p = 0;
        double st = start[0];
        int h = hi_of[0];
#pragma unroll
        for (int i = 1; i < WALK_BINADES; i++)
            if (i < phases && tg >= start[i]) { p = i; st = start[i]; h = hi_of[i]; }
        const double inv = dpow2(23 - j0 - p);
        plan_find(F, R.table(rr, p), h, st * inv, tg * inv);
        if (tid == 0) { plan_want(F, F.hit); plan_want(F, last); }
        last = F.hit;
        __syncthreads();
    }
    // ties at or above the lowest bin of their binade's stretch: what precedes them in their bins is wanted
    if (tid == 0) {
#pragma unroll
        for (int p = 0; p < WALK_BINADES; p++) {
            const WalkTies *t = R.ties(rr) + p;
            const int n = p < phases ? min(__ldcg(&t->n), TIE_CAP) : 0;
#pragma unroll 4
            for (int i = 0; i < n; i++) {
                const int b = (int)((unsigned int)(__ldcg(&t->key[i]) >> 32) >> BIN_SHIFT);
                if (b >= low_of[p] && b < hi_of[p]) plan_want(F, b);
            }
        }
        WalkPicks *o = R.picks(rr);
#pragma unroll 1
        for (int i = 0; i < F.n; i++) { o->bin[i] = F.pick[i]; o->cnt[i] = 0; }
        o->n = F.n;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(SPAN_THREADS, 4) tile_walk_kernel(const __grid_constant__ RowsArgs R) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WalkTileShared *S = reinterpret_cast<WalkTileShared *>(smem_raw);
    __shared__ int S_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_next();
    pdl_wait();
    // A block takes neighbouring spans of the queue's rows, as many as make one round of blocks, and adds up the tables of each
    // row among them once. (Equal shares of every row are not equal shares of the queue: 200 rows of 50257 that sort nothing made 600 of
    // three spans and fewer for 592 blocks, 149 us where this takes 146.) Spans of rows of up to three go one by one: 256 rows
    // of 20000 116 and 113.
    const int total = R.queue[0] * R.nspan;
    if ((int)blockIdx.x >= total) return;
    const bool single = R.nspan < 4;
    const int each = single ? 1 : (total + (int)gridDim.x - 1) / (int)gridDim.x, w0 = blockIdx.x * each, end = single ? total : min(total, w0 + each);
#pragma unroll 1
    for (int w = w0; w < end; w = single ? w + (int)gridDim.x : min(end, (w / R.nspan + 1) * R.nspan)) {
        const int qi = w / R.nspan, rr = R.queue[1 + qi], span0 = w - qi * R.nspan, span1 = single ? span0 + 1 : min(R.nspan, span0 + end - w);
        RowHead *head = R.head(rr);
        const int state = head->state;
        if (state != ST_HEAD && state != ST_PURE) continue;
        const float Z = head->Z, yZ = __fdiv_rn(1.0f, Z);
        const unsigned int tau = head->plan.tau_bits;
        const float hs = head->head_s;
        const int j0 = hs > 0.0f ? fexpo(hs) : 0, nb = (hs > 0.0f && j0 >= -30 && j0 < 0) ? min(WALK_BINADES, -j0) : 0;
        __syncthreads();
        if (state == ST_HEAD) {
#pragma unroll 1
            for (int i = tid; i < nb * NBINS; i += SPAN_THREADS) { (&S->hq[0][0])[i] = 0u; (&S->hqh[0][0])[i] = 0u; }
            __syncthreads();
        }
#pragma unroll 1
        for (int span = span0; span < span1; span++) {
        const int tile = span * (SPAN / TILE) + warp;
        const size_t gt = (size_t)rr * R.ntile + tile;
        const int n = tile < R.ntile ? (int)R.to(rr)[tile].cnt : 0;
        float4 *src = reinterpret_cast<float4 *>(R.elist + gt * TILE);
        if (state == ST_PURE) {
            if (tile >= R.ntile) continue;
            float *list = S->x + (size_t)warp * 32 * PITCH;
            __syncwarp();
            const float est = R.tp[gt].est * yZ;
            QuickSum qs(est, (tile + 1 < R.ntile ? R.tp[gt + 1].est : R.tp[gt].est) * yZ);
            float4 nx = 4 * lane < n ? src[lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
            for (int e0 = 4 * lane; e0 < n; e0 += 128) {
                const float4 v = nx;
                if (e0 + 128 < n) nx = src[(e0 >> 2) + 32];
                float p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    p[u] = e0 + u < n ? prob_of(p[u], Z, yZ) : 0.0f;
                    list[skew(e0 + u)] = p[u];
                    qs.add(p[u]);
                }
                src[e0 >> 2] = make_float4(p[0], p[1], p[2], p[3]);
            }
            __syncwarp();
            if (qs.holds(est)) {
                if (lane == 0) {
                    unsigned int i0 = 0u;
                    const bool item = qs.counts(est, tile, head->plan.top);
                    if (item) { i0 = (unsigned int)atomicAdd(&head->nitem, 1); R.items(rr)[i0] = run_item(qs.k, qs.j, tile, n, 0, 0); }
                    R.to(rr)[tile].ioff = i0; R.to(rr)[tile].nitem = item ? 1 : 0;
                }
                __syncwarp();
                continue;
            }
            const TileChunk ch = tile_chunk(list, n);
            bool care;
            int my_place, c0 = CARE_PLACES;
            unsigned int i0 = 0;
            const int ni = tile_items(list, ch, est, tile, head->plan.top,
                [&](int k, int nc) -> Item * {
                    if (lane == 0) { i0 = (unsigned int)atomicAdd(&head->nitem, k); if (nc) c0 = atomicAdd(&head->ncare, nc); }
                    i0 = __shfl_sync(0xffffffffu, i0, 0); c0 = __shfl_sync(0xffffffffu, c0, 0);
                    return R.items(rr) + i0;
                },
                [&](int i) { return c0 + i < CARE_PLACES ? c0 + i : 255; }, care, my_place);
            store_care(R.care(rr), list, ch, my_place);
            if (lane == 0) { R.to(rr)[tile].ioff = i0; R.to(rr)[tile].nitem = (unsigned short)ni; }
            __syncwarp();
            continue;
        }
        // ---- past a sorted head: what it took is consumed
        float4 nx = 4 * lane < n ? src[lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
        for (int e0 = 4 * lane; e0 < n; e0 += 128) {
            const float4 v = nx;
            if (e0 + 128 < n) nx = src[(e0 >> 2) + 32];
            float p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                p[u] = (e0 + u < n && __float_as_uint(p[u]) < tau) ? prob_of(p[u], Z, yZ) : 0.0f;
                const unsigned int pb = __float_as_uint(p[u]);
                const int bin = (int)(pb >> BIN_SHIFT);
#pragma unroll
                for (int b = 0; b < WALK_BINADES; b++) {
                    const float half = fpow2(j0 + b - 24);   // below half a unit of a binade: adds nothing there, nor in the ones above
                    if (b >= nb || !(p[u] >= half)) break;
                    const float Cm = __fmul_rn(1.5f, fpow2(j0 + b));
                    const float tq = __fadd_rn(p[u], Cm);
                    const float rr_ = __fsub_rn(p[u], __fsub_rn(tq, Cm));
                    if (fabsf(rr_) == half || p[u] >= fpow2(j0 + b - 1)) {
                        // a rounding tie: listed (an element of a quarter of the sum cannot follow a whole head)
                        WalkTies *t = R.ties(rr) + b;
                        const int at = atomicAdd(&t->n, 1);
                        if (at < TIE_CAP) t->key[at] = make_key(pb, tile * TILE + e0 + u);
                        continue;
                    }
                    // p + Cm stays in Cm's binade, whose unit is the sum's: the difference of the two bit
                    // patterns is the count of units
                    const unsigned int qu = __float_as_uint(tq) - __float_as_uint(Cm);
                    if (qu & MASS_LO_MASK) sred_add(&S->hq[b][bin], qu & MASS_LO_MASK);
                    if (qu >> MASS_SPLIT) sred_add(&S->hqh[b][bin], qu >> MASS_SPLIT);
                }
            }
            src[e0 >> 2] = make_float4(p[0], p[1], p[2], p[3]);
        }
        }
        if (state == ST_PURE) continue;
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < nb * NBINS; i += SPAN_THREADS) {
            const unsigned long long q = (unsigned long long)(&S->hq[0][0])[i] + ((unsigned long long)(&S->hqh[0][0])[i] << MASS_SPLIT);
            if (q) atomicAdd(R.table(rr, 0) + i, q);
        }
        // the block that finishes a row's tables works out which bins the walk will want
        __threadfence();
        __syncthreads();
        if (tid == 0) S_last = atomicAdd(&R.picks(rr)->arrived, 1) == (qi * R.nspan + R.nspan - 1) / each - qi * R.nspan / each ? 1 : 0;
        __syncthreads();
        if (S_last && nb > 0) {
            __threadfence();
            plan_picks(R, rr, hs, j0, nb);
        }
    }
}

// =============================================================================
// Kernel 6: the elements of the wanted bins of every walk, gathered over the whole chip. Bound: one pass
// over the lists of queued rows in L2 (12 us for 20 rows of 151936, 3 with none).
// =============================================================================
__global__ void __launch_bounds__(SPAN_THREADS, 4) tile_pick_kernel(const __grid_constant__ RowsArgs R) {
    __shared__ unsigned char slot[NBINS];   // 0: not wanted
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_next();
    pdl_wait();
    const int work = R.queue[0] * R.nspan;
#pragma unroll 1
    for (int wi = blockIdx.x; wi < work; wi += gridDim.x) {
        const int rr = R.queue[1 + wi / R.nspan], span = wi % R.nspan, tile = span * (SPAN / TILE) + warp;
        if (R.head(rr)->state != ST_HEAD) continue;
        WalkPicks *pk = R.picks(rr);
        const int npick = pk->n;
        if (npick == 0) continue;
        const int n = tile < R.ntile ? (int)R.to(rr)[tile].cnt : 0;
        const uint4 *src = reinterpret_cast<const uint4 *>(R.elist + ((size_t)rr * R.ntile + tile) * TILE);
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (4 * (lane + 32 * i) < n) v[i] = src[lane + 32 * i];
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < NBINS / 4; i += SPAN_THREADS) reinterpret_cast<unsigned int *>(slot)[i] = 0u;
        __syncthreads();
        if (tid < npick) slot[pk->bin[tid]] = (unsigned char)(tid + 1);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int e0 = 4 * (lane + 32 * i);
            if (e0 >= n) continue;
            const unsigned int p[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (e0 + u >= n || p[u] == 0u) continue;
                const int k = slot[p[u] >> BIN_SHIFT];
                if (k) {
                    const int at = atomicAdd(&pk->cnt[k - 1], 1);
                    if (at < PICK_CAP) R.picked(rr, k - 1)[at] = make_key(p[u], tile * TILE + e0 + u);
                }
            }
        }
    }
}

// =============================================================================
// Kernel 7: the rows that were queued, one block each: the general forms of everything kernel 4 does, and
// what it does not. Bound: latency of code that runs once and of one warp's dependent additions: 24 us where
// nothing is sorted, 39 for 58 walks past the head, 200 for a row with more careful chunks than kernel 4 takes.
// =============================================================================
struct __align__(16) AuxF {
    union {
        float tile[NWARP * 32 * PITCH];    // tiles being worked on, one per warp (a span and its scratch use the same space)
        struct {
            union {
                struct { unsigned int hq[NBINS], hqh[NBINS], hc[NBINS]; } h;
            } u;
            unsigned long long cand[NC];   // the head's, then a bin's candidates
            unsigned long long tmp[NC];
            unsigned int sbin[NBINS];
            __align__(16) float pc[NC];
            __align__(16) float pre[HEADCAP];
            unsigned int hidx[HEADCAP];
        };
    };
    Item items[ITEM_CAP + 1];
    unsigned int isrc[ITEM_CAP];           // tile << 8 | slot of the fetched entries (255: none)
    __align__(16) float care[CARE_CAP * 32];
    unsigned short careidx[CARE_CAP];
    __align__(16) float ebuf[TILE];
    unsigned short tcnt[MAX_TILES];        // entries in the tile's list
    unsigned short tni[MAX_TILES];         // items of the tile
    int toff[MAX_TILES + 1];               // first item of the tile
    unsigned int tio[MAX_TILES];           // where its items begin
    float tsum[MAX_TILES];
    double wsd[2 * (NWARP + 1)];
    unsigned long long wsu[NWARP + 1];
    float wsf[NWARP + 1];
    int wsi[NWARP + 1];
    int ncand, ncare, evt_thread, specbin, hit_bin;
    unsigned long long hit_qbefore, hit_cbefore, tot_q, tot_c;
    float b_s; int b_event; int b_idx; float b_p; long long b_pos; int b_aux;
    float b_sum, b_target;
    unsigned int w_sb; int w_i, w_need, w_found, w_tile, w_at;   // the items' runner
    WalkTies ties[WALK_BINADES]; WalkPicks picks;   // row_tail's copies
    int ntie; unsigned long long tkey[TIE_CAP]; int tbin[TIE_CAP]; unsigned char tord[TIE_CAP]; unsigned int tpq_lo[TIE_CAP], tpq_hi[TIE_CAP];
    unsigned long long tpqm[TIE_CAP], tabove[TIE_CAP], tc[TIE_CAP];
    unsigned int tbits[NBINS / 32];
};
static_assert(sizeof(SpanScratch) + (size_t)SPAN_THREADS * PITCH * 4 <= sizeof(float) * NWARP * 32 * PITCH, "a span and its scratch fit the tiles' space");

// Profiling stamps exist in the testing build only (per row 32 slots of clock readings and counts).
#ifdef MOLLA_SAMPLE_TESTING
#define FSTAMP(i) do { if (c.R->a.prof && c.tid == 0) c.R->a.prof[(long long)c.r * 32 + (i)] = clock64(); } while (0)
#define FCOUNT(i, v) do { if (c.R->a.prof && c.tid == 0) c.R->a.prof[(long long)c.r * 32 + (i)] += (v); } while (0)
#else
#define FSTAMP(i) do { } while (0)
#define FCOUNT(i, v) do { } while (0)
#endif

struct CtxF {
    int tid, lane, warp;
    AuxF *A;
    unsigned int status;
    const RowsArgs *R;
    int rr, r;
    RowCfg cfg;
    RowPlan pl;
    int tj0, tnb;                // binades that tile_walk has left tables for
    int npick;                   // bins that tile_pick has gathered
    bool first_table;            // the table of binade tj0 is in shared memory
    float *list;                 // this row's [ntile][TILE]
    Item *gitems;                // this row's items
    const unsigned int *kmask;   // this row's [ntile][32]
};

// One entry of the list, as a token id: the nth logit its tile kept.
__device__ __noinline__ int token_of(const CtxF &c, int tile, int nth) {
    const unsigned int *m = c.kmask + (size_t)tile * 32;
#pragma unroll 8
    for (int g = 0; g < 32; g++) {
        unsigned int w = m[g];
        const int n = __popc(w);
        if (nth >= n) { nth -= n; continue; }
        while (nth-- > 0) w &= w - 1u;
        return tile * TILE + g * 32 + __ffs((int)w) - 1;
    }
    return tile * TILE;
}
__device__ __forceinline__ int token_of(const CtxF &c, int pos) { return token_of(c, pos >> 10, pos & (TILE - 1)); }

// Tiles [t0, t1) of one span evaluated again, as kernel 3 did it: their values packed into dst or the list.
__device__ __noinline__ void tile_again(CtxF &c, int t0, int t1, float *dst, bool to_list) {
    AuxF *A = c.A;
    IN_SHARED(A);
    const RowsArgs &R = *c.R;
    const int span = t0 / (SPAN / TILE);
    SpanScratch *s = reinterpret_cast<SpanScratch *>(A->tile + SPAN_THREADS * PITCH);
    __syncthreads();
    if (c.tid < SPAN_THREADS) span_fetch(R.a, c.cfg.lrow, span * SPAN, A->tile);
    span_ready(R.a, c.cfg, c.r, span * SPAN, A->tile, s, c.tid < SPAN_THREADS);
    const int t = span * (SPAN / TILE) + c.warp;
    if (c.warp < SPAN / TILE && t >= t0 && t < t1) {
        const float thr = R.tp[(size_t)c.rr * R.ntile + t].thr;
        float *list = A->tile + (size_t)c.warp * 32 * PITCH;
        const TileEval e = tile_eval(list, reinterpret_cast<unsigned short *>(s->cnt) + c.warp * TILE, thr, c.cfg.T, __fdiv_rn(1.0f, c.cfg.T), c.pl.top,
                                     (c.pl.flags & F_FASTDIV) && thr > -INFINITY, [](unsigned int, bool, unsigned int) {});
        float *to = to_list ? c.list + (size_t)t * TILE : dst;
#pragma unroll 1
        for (int i = c.lane; i < (to_list ? e.total : TILE); i += 32) to[i] = i < e.total ? list[skew(i)] : 0.0f;
        if (to_list) {
            const_cast<unsigned int *>(c.kmask)[(size_t)t * 32 + c.lane] = e.keep;
            if (c.lane == 0) A->tcnt[t] = (unsigned short)e.total;   // (kernel 3 need not have counted them)
        }
    }
    __syncthreads();
}

// n values, four at a time from a 16-byte aligned place that is padded with zeros, added one by one to
// the sum with bit pattern `sb`. Every lane of the warp does the same. With `locate`, stops at the first
// value behind which the sum exceeds `target`; returns its number, or -1.
__device__ __forceinline__ int run_values(unsigned int &sb, const float *v, int n, bool locate, float target) {
    const float4 *v4 = reinterpret_cast<const float4 *>(v);
    float s = __uint_as_float(sb);
#pragma unroll 1
    for (int i = 0; i < n; i += 8) {
        const float4 x = v4[i >> 2], y = v4[(i >> 2) + 1];
        const float s0 = s;
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, x.x), x.y), x.z), x.w);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, y.x), y.y), y.z), y.w);
        if (locate && target < s) {
            s = s0;
#pragma unroll 1
            for (int u = 0; u < 8; u++) {
                s = __fadd_rn(s, v[i + u]);
                if (target < s) { sb = __float_as_uint(s); return i + u; }
            }
        }
    }
    sb = __float_as_uint(s);
    return -1;
}

// One warp: the items of the batch in shared memory from A->w_i on, 32 at a time. Runs in the sum's
// binade are consumed by a scan of their units, whatever needs care one by one. Ends with A->w_need = -1
// (the batch is through, or the target is found) or the item whose values are wanted.
__device__ void run_items(AuxF *A, int n, bool locate, float target) {
    IN_SHARED(A);
    const int lane = threadIdx.x & 31;
    unsigned int sb = A->w_sb;
    int i = A->w_found ? n : A->w_i, need = -1;
    bool found = false;
    while (i < n && need < 0 && !found) {
        const int i0 = i;
        Item it;
        it.ka = 0u; it.kb = 0u; it.meta = 0u; it.oc = 0u;
        if (i0 + lane < n) it = A->items[i0 + lane];
        const unsigned int jb = it.jb(), kind = it.kind();
        const bool plain = i0 + lane < n && kind == K_RUN && parity_free(it.ka);
        const unsigned int incl = warp_incl_scan(plain ? it.ka : 0u, lane);
        int at = 0;
        unsigned int base = 0u;      // units of the runs before `at`
        while (at < 32 && i0 + at < n && need < 0 && !found) {
            const unsigned int j = sb >> 23, to = sb + (incl - base);
            const bool fits = plain && jb == j && (to >> 23) == j && !(locate && target < __uint_as_float(to));
            const unsigned int stop = ~__ballot_sync(0xffffffffu, fits) & ~((1u << at) - 1u);
            const int f = stop ? __ffs((int)stop) - 1 : 32;
            if (f > at) { sb = __shfl_sync(0xffffffffu, to, f - 1); at = f; }
            if (at >= 32 || i0 + at >= n) break;
            const unsigned int ka = __shfl_sync(0xffffffffu, it.ka, at), kb = __shfl_sync(0xffffffffu, it.kb, at);
            const unsigned int meta = __shfl_sync(0xffffffffu, it.meta, at), oc = __shfl_sync(0xffffffffu, it.oc, at);
            base = __shfl_sync(0xffffffffu, incl, at);
            const unsigned int kd = (meta >> 8) & 3u, jx = meta & 0xffu, e = sb >> 23;
            bool ok = false;
            unsigned int nx = sb;
            if (kd != K_STEP) {
                if (e == jx) { nx = sb + units(ka, sb); ok = (nx >> 23) == e; }
                else if (kd == K_DUAL && e == jx + 1u) { nx = sb + units(kb, sb); ok = (nx >> 23) == e; }
            }
            if (ok && !(locate && target < __uint_as_float(nx))) { sb = nx; at++; continue; }
            const unsigned int src = A->isrc[i0 + at];
            if ((src & 0xffu) == 255u) { need = i0 + at; break; }
            const int hit = run_values(sb, A->care + (src & 0xffu) * 32, (int)(oc & 0x7ffu), locate, target);
            at++;
            if (hit >= 0) {
                found = true;
                if (lane == 0) { A->w_found = 1; A->w_tile = (int)(src >> 8); A->w_at = (int)((oc >> 11) & 0x3ffu) + hit; }
            }
        }
        i = i0 + at;
    }
    if (lane == 0) { A->w_sb = sb; A->w_i = i; A->w_need = need; }
}

// The exact sequential fp32 sum over the row's items (A->tni of each tile in the row's item space).
// Returns it; with `locate`, A->w_found says whether the running sum exceeded `target` and A->w_tile,
// A->w_at at which list entry.
__device__ __noinline__ float exact_sum(CtxF &c, bool locate, float target) {
    AuxF *A = c.A;
    IN_SHARED(A);
    const RowsArgs &R = *c.R;
    __syncthreads();
    int total;
    {
        const int t = 2 * c.tid;
        const int n0 = t < R.ntile ? A->tni[t] : 0, n1 = t + 1 < R.ntile ? A->tni[t + 1] : 0;
        const int ex = block_excl_scan<int>(n0 + n1, A->wsi, &total);
        if (t < R.ntile) A->toff[t] = ex;
        if (t + 1 < R.ntile) A->toff[t + 1] = ex + n0;
    }
    if (c.tid == 0) { A->w_sb = 0u; A->w_found = 0; A->w_tile = 0; A->w_at = 0; }
#pragma unroll 1
    for (int b0 = 0; b0 < total; b0 += ITEM_CAP) {
        const int n = min(ITEM_CAP, total - b0);
        __syncthreads();
        if (c.tid == 0) { A->ncare = 0; A->w_i = 0; }
        __syncthreads();
        // an item per thread: its tile is found in the tiles' offsets
#pragma unroll 1
        for (int i = c.tid; i < n; i += NT) {
            int lo = 0, hi = R.ntile - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (A->toff[mid] <= b0 + i) lo = mid; else hi = mid - 1;
            }
            const Item it = c.gitems[A->tio[lo] + (b0 + i - A->toff[lo])];
            unsigned int slot = 255u;
            if (it.kind() != K_RUN && it.cnt() <= 32) {
                const int q = satom_add(&A->ncare, 1);
                if (q < CARE_CAP) { slot = (unsigned int)q; A->careidx[q] = (unsigned short)i; }
            }
            A->items[i] = it;
            A->isrc[i] = ((unsigned int)lo << 8) | slot;
        }
        __syncthreads();
        const int ncare = min(A->ncare, CARE_CAP);
#pragma unroll 1
        for (int q = c.warp; q < ncare; q += NWARP) {
            const int i = A->careidx[q];
            const Item it = A->items[i];
            A->care[q * 32 + c.lane] = c.lane >= it.cnt() ? 0.0f : (it.place() != 255u ? R.care(c.rr)[it.place() * 32 + c.lane] : c.list[(size_t)it.tile() * TILE + it.off() + c.lane]);
        }
        FCOUNT(20, n); FCOUNT(21, ncare); if (!locate) FSTAMP(2);
#pragma unroll 1
        for (int round = 0; round <= n; round++) {   // (each round but the last is for one more item)
            __syncthreads();
            if (c.warp == 0) run_items(A, n, locate, target);
            __syncthreads();
            const int want = A->w_need;
            if (want < 0 || A->w_found) break;
            // a run whose guess was wrong, or that holds the target: its values, one by one
            const Item it = A->items[want];
            const int t = it.tile(), off = it.off(), m = it.cnt();
            FCOUNT(23, 1);
            if (it.place() != 255u) {
                if (c.tid < 32) A->ebuf[c.tid] = c.tid < m ? R.care(c.rr)[it.place() * 32 + c.tid] : 0.0f;
            } else if ((c.pl.flags & F_LIST) || it.kind() != K_RUN) {
#pragma unroll 1
                for (int i = c.tid; i < ((m + 7) & ~7); i += NT) A->ebuf[i] = i < m ? c.list[(size_t)t * TILE + off + i] : 0.0f;
            } else {
                tile_again(c, t, t + 1, A->ebuf, false);
                float x[TILE / NT];
#pragma unroll 1
                for (int i = c.tid, u = 0; u < TILE / NT; i += NT, u++) x[u] = i < m ? A->ebuf[off + i] : 0.0f;
                __syncthreads();
#pragma unroll 1
                for (int i = c.tid, u = 0; u < TILE / NT; i += NT, u++) A->ebuf[i] = x[u];
            }
            __syncthreads();
            if (c.warp == 0) {
                unsigned int sb = A->w_sb;
                const int hit = run_values(sb, A->ebuf, m, locate, target);
                if (c.lane == 0) {
                    A->w_sb = sb; A->w_i = want + 1;
                    if (hit >= 0) { A->w_found = 1; A->w_tile = t; A->w_at = off + hit; }
                }
            }
        }
        if (A->w_found) break;
    }
    __syncthreads();
    return __uint_as_float(A->w_sb);
}

// Calls f(values, position of the first, where they are) for the row's list, four neighbouring entries of
// a lane at a time (zero: none). All lanes of a warp make the same calls. (Kept small: it is rarely needed, and cold code
// is fetched from L2.)
template <class F>
__device__ __forceinline__ void for_list4(const CtxF &c, F f) {
    const AuxF *A = c.A;
    IN_SHARED(A);
#pragma unroll 1
    for (int t = c.warp; t < c.R->ntile; t += NWARP) {
        const int n = A->tcnt[t];
        const uint4 *src = reinterpret_cast<const uint4 *>(c.list + (size_t)t * TILE) + c.lane;
        uint4 nx = make_uint4(0u, 0u, 0u, 0u);
        if (4 * c.lane < n) nx = src[0];
#pragma unroll 1
        for (int i = 0; 128 * i < n; i++) {
            const uint4 v = nx;
            const int e0 = 4 * (c.lane + 32 * i);
            if (e0 + 128 < n) nx = src[32 * (i + 1)];
            const unsigned int eb[4] = {e0 < n ? v.x : 0u, e0 + 1 < n ? v.y : 0u, e0 + 2 < n ? v.z : 0u, e0 + 3 < n ? v.w : 0u};
            f(eb, t * TILE + e0, c.list + (size_t)t * TILE + e0);
        }
    }
}

__device__ __noinline__ void sort_head(CtxF &c, int n) {
    AuxF *A = c.A;
    IN_SHARED(A);
    static_assert(HEADCAP <= NC, "the sorted keys fit the candidates' space");
    __syncthreads();
    sort_keys<NT, 96>(n, A->cand, A->tmp, A->pc, A->sbin, reinterpret_cast<unsigned int *>(A->wsi), reinterpret_cast<unsigned int *>(A->wsf));
}

// More candidates than the head holds (few lanes for a wide top-k, or many equal values): a finer
// edge from the values themselves. Returns the number of candidates written to `cand` and moves the
// row's edge up, or a number above HEADCAP where one bin of values alone is too full.
__device__ __noinline__ int narrow_head(CtxF &c, unsigned long long *cand) {
    AuxF *A = c.A;
    IN_SHARED(A);
    __syncthreads();
#pragma unroll 1
    for (int i = c.tid; i < NBINS; i += NT) A->u.h.hc[i] = 0u;
    if (c.tid == 0) { A->ncand = 0; A->evt_thread = -1; }
    __syncthreads();
    for_list4(c, [&](const unsigned int (&eb)[4], int, float *) {
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (eb[u]) sred_add(&A->u.h.hc[eb[u] >> BIN_SHIFT], 1u);
    });
    __syncthreads();
    int n[BPT], sum = 0, tot;
#pragma unroll
    for (int i = 0; i < BPT; i++) { n[i] = (int)A->u.h.hc[NBINS - 1 - BPT * c.tid - i]; sum += n[i]; }
    int run = block_excl_scan<int>(sum, A->wsi, &tot);
    const int need = min(c.pl.need, tot);
#pragma unroll
    for (int i = 0; i < BPT; i++) {
        if (run < need && run + n[i] >= need) { A->evt_thread = NBINS - 1 - BPT * c.tid - i; A->b_idx = run + n[i]; }
        run += n[i];
    }
    __syncthreads();
    if (A->evt_thread < 0 || A->b_idx > HEADCAP) return HEADCAP + 1;
    const unsigned int edge = (unsigned int)A->evt_thread << BIN_SHIFT;
    c.pl.tau_bits = edge > 1u ? edge : 1u;
#pragma unroll 1
    for (int t = c.warp; t < c.R->ntile; t += NWARP) {
        unsigned int m = c.kmask[(size_t)t * 32 + c.lane];
        const float *src = c.list + (size_t)t * TILE + (warp_incl_scan(__popc(m), c.lane) - __popc(m));
#pragma unroll 1
        for (int i = 0; m; i++, m &= m - 1u) {
            const unsigned int eb = __float_as_uint(src[i]);
            if (eb >= c.pl.tau_bits) cand[satom_add(&A->ncand, 1)] = make_key(eb, t * TILE + c.lane * 32 + __ffs((int)m) - 1);
        }
    }
    __syncthreads();
    return A->ncand;
}

// The descending walk past the sorted head (sample.mojo:492-506 and :580-590) over the row's list of
// probabilities. State: exact running sum, elements consumed, and tau: everything with probability
// bits >= tau is consumed. Every phase histograms what remains by value bin, consumes whole bins up
// to the first one holding an event, gathers that bin, sorts it and adds it element by element.
//
// An element whose addition would be a rounding tie (its value is an odd multiple of half the
// running sum's unit) rounds up or down with the parity of the sum before it. Such elements do
// not stop a phase: they are listed, a second pass adds up what precedes each of them inside
// its own bin, and one thread then resolves them from the top down, each from the exact integer
// sum before it; their contributions go into their bins' masses before the event is searched.
struct FWalk {
    float s; long long pos; unsigned int tau;
    int event; int idx; float p; int tie;   // idx: position in the list, or (crowded) the same
};
// Where a walk's last phase began. The draw walk adds up the same elements in the same order as
// the cut walk before it, so when its target is not reached before that point it starts there,
// on the bin tables that are still standing, and skips the passes that built them.
struct FResume {
    int valid;
    float s; long long pos; unsigned int tau;
    int lvl; unsigned int lo; int shift; int tie_mode; int ntie; int tabbed;
};

// position of the (nth+1)-th entry, in vocabulary order, whose bits equal `eb`
__device__ __noinline__ int list_nth_equal(CtxF &c, unsigned int eb, int nth) {
    AuxF *A = c.A;
    IN_SHARED(A);
    __syncthreads();
#pragma unroll 1
    for (int t = c.warp; t < c.R->ntile; t += NWARP) {
        int n = 0;
#pragma unroll 1
        for (int i = c.lane; i < A->tcnt[t]; i += 32) n += __float_as_uint(c.list[(size_t)t * TILE + i]) == eb ? 1 : 0;
        n = __reduce_add_sync(0xffffffffu, n);
        if (c.lane == 0) A->toff[t] = n;
    }
    __syncthreads();
    if (c.tid == 0) {
        int seen = 0, at = 0;
#pragma unroll 1
        for (int t = 0; t < c.R->ntile; t++) {
            if (nth < seen + A->toff[t]) {
#pragma unroll 1
                for (int i = 0; i < A->tcnt[t]; i++)
                    if (__float_as_uint(c.list[(size_t)t * TILE + i]) == eb && seen++ == nth) { at = t * TILE + i; break; }
                break;
            }
            seen += A->toff[t];
        }
        A->b_idx = at;
    }
    __syncthreads();
    return A->b_idx;
}

__device__ __noinline__ void descend_list(CtxF &c, FWalk &w, float x_ge, float x_gt, long long nstop, FResume &rs, bool try_resume) {
    AuxF *A = c.A;
    IN_SHARED(A);
    const bool counting = nstop >= 0;
    int lvl = 1;
    unsigned int lo = 0u;
    int shift = BIN_SHIFT;
    bool tie_mode = true;
    const bool resumed = try_resume && rs.valid && !counting && x_ge >= 3.0e38f && !(x_gt < rs.s);
    if (resumed) {
        w.s = rs.s; w.pos = rs.pos; w.tau = rs.tau;
        lvl = rs.lvl; lo = rs.lo; shift = rs.shift; tie_mode = rs.tie_mode != 0;
    }
#pragma unroll 1
    for (int phase = 0; phase < 8192; phase++) {
        FCOUNT(22, 1);
        const bool reuse = resumed && phase == 0 && !rs.tabbed;  // this phase's tables stand already
        __syncthreads();
        const bool have_s = w.s > 0.0f;
        const int j = have_s ? fexpo(w.s) : 0;
        const bool binade_ok = have_s && j >= -100 && j <= 100;
        const float Cm = __fmul_rn(1.5f, fpow2(j)), halfu = fpow2(j - 24), bigthr = fpow2(j - 1);
        const float inv_u = fpow2(23 - j);
        const unsigned int cm_bits = __float_as_uint(Cm);
        const bool ties_listed = tie_mode && lvl == 1 && binade_ok;
        const unsigned int wtau = w.tau;
        // tile_walk's tables hold whole bins: they serve while what is consumed ends at a bin's edge (not where the walk before has left
        // its own, with its ties and what precedes each of them)
        const WalkTies *tt = nullptr;
        const unsigned long long *tab = nullptr;
        int bin_hi = NBINS;
        if (!reuse && c.tnb > 0 && ties_listed && !counting && j >= c.tj0 && j < c.tj0 + c.tnb && (wtau == 0xFFFFFFFFu || (wtau & ((1u << BIN_SHIFT) - 1u)) == 0u)) {
            tt = A->ties + (j - c.tj0);
            if (tt->n <= TIE_CAP) {
                tab = (j == c.tj0 && c.first_table) ? reinterpret_cast<const unsigned long long *>(&A->u.h) : c.R->table(c.rr, j - c.tj0);
                if (wtau != 0xFFFFFFFFu) bin_hi = (int)(wtau >> BIN_SHIFT);
            }
        }
        const bool tabbed = tab != nullptr;
        if (!reuse) {
            if (!tabbed) c.first_table = false;
            if (!tabbed)
#pragma unroll 1
                for (int i = c.tid; i < NBINS; i += NT) { A->u.h.hq[i] = 0u; A->u.h.hqh[i] = 0u; A->u.h.hc[i] = 0u; }
#pragma unroll 1
            for (int i = c.tid; i < NBINS / 32; i += NT) A->tbits[i] = 0u;
            rs.valid = 1; rs.s = w.s; rs.pos = w.pos; rs.tau = w.tau;
            rs.lvl = lvl; rs.lo = lo; rs.shift = shift; rs.tie_mode = tie_mode ? 1 : 0; rs.ntie = 0; rs.tabbed = tabbed ? 1 : 0;
        }
        if (c.tid == 0) {
            if (!reuse) A->specbin = -1;
            A->ncand = 0; A->ntie = 0;
        }
        __syncthreads();
        BinQuery qy;
        qy.bin_hi = bin_hi; qy.spec_bits = nullptr; qy.specbin = -1;
        qy.hq = A->u.h.hq; qy.hqh = A->u.h.hqh; qy.hc = A->u.h.hc;
        qy.pos0 = (unsigned long long)w.pos;
        qy.nstop = counting ? (unsigned long long)nstop : ~0ull;
        qy.counts = counting || !binade_ok;
        qy.m0 = 0; qy.xq = ~0ull;
        if (binade_ok) {
            qy.m0 = (unsigned long long)((double)w.s * (double)inv_u);
            unsigned long long xq = 1ull << 24;  // leaving the binade
            if (x_ge < 3.0e38f) {
                double t = ceil((double)x_ge * (double)inv_u);
                if (t < (double)xq) xq = (t <= 0.0) ? 0ull : (unsigned long long)t;
            }
            if (x_gt < 3.0e38f) {
                double t = floor((double)x_gt * (double)inv_u) + 1.0;
                if (t < (double)xq) xq = (t <= 0.0) ? 0ull : (unsigned long long)t;
            }
            qy.xq = xq;
        } else {
            qy.pos0 = 0; qy.nstop = 1;  // nothing consumed yet: take the highest non-empty bin
        }
        auto bin_load = [&](int b, unsigned long long &q, unsigned long long &n) {
            if (tabbed) { q = tab[b]; n = 0ull; return; }
            q = (unsigned long long)qy.hq[b] + ((unsigned long long)qy.hqh[b] << MASS_SPLIT);
            n = qy.hc[b];
        };
        int ntie = rs.ntie;
        bool searched = false;
        if (tabbed) {
            // without the ties first: they only add, so the event lies in the bin found here or in a higher
            // one, and a tie below that bin changes nothing
            find_event_bin_with(c, qy, bin_load);
            const int b0 = A->hit_bin;
            if (c.tid < tt->n) {
                const unsigned long long key = tt->key[c.tid];
                const int b = (int)((unsigned int)(key >> 32) >> BIN_SHIFT);
                if (b < bin_hi && b >= b0) { const int at = satom_add(&A->ntie, 1); A->tkey[at] = key; A->tbin[at] = b; }
            }
            __syncthreads();
            ntie = A->ntie;
            rs.ntie = ntie;
            searched = ntie == 0;
        } else if (!reuse) {
            const bool count_all = counting || !binade_ok;
            for_list4(c, [&](const unsigned int (&ebs)[4], int pos0, float *) {
                bool rare = false;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned int eb = ebs[u];
                    const bool live = eb != 0u && eb < wtau && eb >= lo;
                    const int bin = (int)((eb - lo) >> shift);
                    const float p = __uint_as_float(eb);
                    const float tq = __fadd_rn(p, Cm);
                    const float rr = __fsub_rn(p, __fsub_rn(tq, Cm));
                    const bool special = (fabsf(rr) == halfu) || (p >= bigthr);
                    // below bigthr, p + Cm stays in Cm's binade, whose unit is the sum's: the difference
                    // of the two bit patterns is the count of units
                    const unsigned int qu = __float_as_uint(tq) - cm_bits;
                    if (live && count_all) sred_add(&A->u.h.hc[bin], 1u);
                    const bool plain = live && binade_ok && !special;
                    if (plain && (qu & MASS_LO_MASK)) sred_add(&A->u.h.hq[bin], qu & MASS_LO_MASK);
                    if (plain && (qu >> MASS_SPLIT)) sred_add(&A->u.h.hqh[bin], qu >> MASS_SPLIT);
                    rare |= live && binade_ok && special;
                }
                if (__any_sync(0xffffffffu, rare)) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const unsigned int eb = ebs[u];
                        if (!(eb != 0u && eb < wtau && eb >= lo)) continue;
                        const int bin = (int)((eb - lo) >> shift);
                        const float p = __uint_as_float(eb);
                        const float q = __fsub_rn(__fadd_rn(p, Cm), Cm);
                        const bool tie = fabsf(__fsub_rn(p, q)) == halfu;
                        if ((p >= bigthr) || (tie && !ties_listed)) { sred_max(&A->specbin, bin); continue; }
                        if (tie) {
                            const int pos = satom_add(&A->ntie, 1);
                            if (pos < TIE_CAP) { A->tkey[pos] = make_key(eb, pos0 + u); A->tbin[pos] = bin; }
                        }
                    }
                }
            });
            __syncthreads();
            ntie = ties_listed ? A->ntie : 0;
            rs.ntie = ntie;
            if (ntie > TIE_CAP) { tie_mode = false; c.status |= MOLLA_ROW_SLOW_PATH; continue; }  // too many: they stop phases instead
        }
        const WalkPicks *pk = &A->picks;
        auto pick_of = [&](int b) -> int {   // the bin's place among the gathered ones, -1: not there
#pragma unroll 1
            for (int i = 0; i < c.npick; i++)
                if (pk->bin[i] == b && pk->cnt[i] <= PICK_CAP) return i;
            return -1;
        };
        if (!reuse && ntie > 0) {
            // what precedes each listed element inside its own bin (descending value, then ascending id)
            if (c.tid < ntie) {
                const int b = A->tbin[c.tid];
                A->tpq_lo[c.tid] = 0u; A->tpq_hi[c.tid] = 0u;
                sred_or(&A->tbits[b >> 5], 1u << (b & 31));
            }
            __syncthreads();
            int tb_lo = NBINS, tb_hi = -1;
#pragma unroll 1
            for (int t = 0; t < ntie; t++) { tb_lo = min(tb_lo, A->tbin[t]); tb_hi = max(tb_hi, A->tbin[t]); }
            const unsigned int tb_span = (unsigned int)(tb_hi - tb_lo);
            bool gathered = tabbed;
#pragma unroll 1
            for (int t = 0; t < ntie && gathered; t++) gathered = pick_of(A->tbin[t]) >= 0;
            if (gathered) {
#pragma unroll 1
                for (int t = 0; t < ntie; t++) {
                    const int k = pick_of(A->tbin[t]), m = pk->cnt[k];
                    const unsigned long long *keys = c.R->picked(c.rr, k), tk = A->tkey[t];
#pragma unroll 1
                    for (int i = c.tid; i < m; i += NT) {
                        const unsigned long long key = keys[i];
                        const unsigned int eb = (unsigned int)(key >> 32);
                        const float p = __uint_as_float(eb);
                        const float tq = __fadd_rn(p, Cm);
                        if (eb >= wtau || !(key > tk) || fabsf(__fsub_rn(p, __fsub_rn(tq, Cm))) == halfu || p >= bigthr) continue;
                        const unsigned int qu = __float_as_uint(tq) - cm_bits;
                        if (qu) {
                            sred_add(&A->tpq_lo[t], qu & MASS_LO_MASK);
                            if (qu >> MASS_SPLIT) sred_add(&A->tpq_hi[t], qu >> MASS_SPLIT);
                        }
                    }
                }
            } else for_list4(c, [&](const unsigned int (&ebs)[4], int pos0, float *) {
                bool near = false;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned int eb = ebs[u];
                    const int bin = (int)((eb - lo) >> shift);
                    near |= eb != 0u && eb < wtau && eb >= lo && (unsigned int)(bin - tb_lo) <= tb_span;
                }
                if (!__any_sync(0xffffffffu, near)) return;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned int eb = ebs[u];
                    if (eb == 0u || eb >= wtau || eb < lo) continue;
                    const int bin = (int)((eb - lo) >> shift);
                    if (!((A->tbits[bin >> 5] >> (bin & 31)) & 1u)) continue;
                    const float p = __uint_as_float(eb);
                    const float tq = __fadd_rn(p, Cm);
                    const float rr = __fsub_rn(p, __fsub_rn(tq, Cm));
                    if (fabsf(rr) == halfu || p >= bigthr) continue;
                    const unsigned int qu = __float_as_uint(tq) - cm_bits;
                    const unsigned long long key = make_key(eb, pos0 + u);
#pragma unroll 1
                    for (int t = 0; t < ntie; t++)
                        if (A->tbin[t] == bin && key > A->tkey[t] && qu) {  // two halves, as in the bin tables
                            sred_add(&A->tpq_lo[t], qu & MASS_LO_MASK);
                            if (qu >> MASS_SPLIT) sred_add(&A->tpq_hi[t], qu >> MASS_SPLIT);
                        }
                }
            });
            __syncthreads();
        }
        if (c.tid < ntie) {
            if (!reuse) A->tpqm[c.tid] = (unsigned long long)A->tpq_lo[c.tid] + ((unsigned long long)A->tpq_hi[c.tid] << MASS_SPLIT);
            A->tc[c.tid] = 0ull;
        }
        __syncthreads();
        if (!tabbed) qy.specbin = A->specbin;
        if (!searched)
        find_event_bin_adj(c, qy, bin_load,
            [&](unsigned long long (&q)[BPT], unsigned long long eq) -> bool {
                if (ntie == 0) return false;
                // the mass before each listed element: the bins above its own (the thread that
                // owns the bin knows), and what precedes it inside the bin
                unsigned long long run = eq;
#pragma unroll
                for (int i = 0; i < BPT; i++) {
                    const int b = NBINS - 1 - BPT * c.tid - i;
#pragma unroll 1
                    for (int t = 0; t < ntie; t++)
                        if (A->tbin[t] == b) A->tabove[t] = run;
                    run += q[i];
                }
                if (c.tid < ntie) {   // the ties' order from the top
                    int rank = 0;
#pragma unroll 1
                    for (int t = 0; t < ntie; t++) rank += A->tkey[t] > A->tkey[c.tid] ? 1 : 0;
                    A->tord[rank] = (unsigned char)c.tid;
                }
                __syncthreads();
                if (c.tid == 0) {
                    // from the top down (what lies below an event never matters: the walk stops there)
                    unsigned long long carried = 0ull;
#pragma unroll 1
                        for (int round = 0; round < ntie; round++) {
                            const int best = A->tord[round];
                            const float p = key_val(A->tkey[best]);
                        const float qf = __fsub_rn(__fadd_rn(p, Cm), Cm);
                        unsigned long long k = (unsigned long long)__float2uint_rn(__fmul_rn(qf, inv_u));
                        if (qf > p) k -= 1ull;  // the multiple of the unit below p
                        const unsigned long long mb = qy.m0 + A->tabove[best] + A->tpqm[best] + carried;
                        if (qy.xq != ~0ull && mb >= qy.xq) break;
                        const unsigned long long ct = k + ((mb + k) & 1ull);
                        A->tc[best] = ct;
                        carried += ct;
                        if (qy.xq != ~0ull && mb + ct >= qy.xq) break;
                    }
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < BPT; i++) {
                    const int b = NBINS - 1 - BPT * c.tid - i;
#pragma unroll 1
                    for (int t = 0; t < ntie; t++)
                        if (A->tbin[t] == b) q[i] += A->tc[t];
                }
                return true;
            });
        if (phase < 2 && !try_resume) FSTAMP(11 + 3 * phase);
        const int hb = A->hit_bin;
        if (hb < 0) {
            // nothing left in this range triggers an event: consume it whole
            if (binade_ok) w.s = (float)((double)(qy.m0 + A->tot_q) * (double)fpow2(j - 23));
            w.pos += (long long)A->tot_c;
            if (lvl == 1) { w.tau = 0; w.event = EV_EXHAUSTED; return; }
            w.tau = lo; lvl = 1; lo = 0u; shift = BIN_SHIFT;  // back to the coarse bins below this range
            continue;
        }
        const unsigned long long qb = A->hit_qbefore, cb = A->hit_cbefore;
        const unsigned int blo = lo + ((unsigned int)hb << shift);
        const unsigned long long bhi64 = (unsigned long long)lo + ((unsigned long long)(hb + 1) << shift);
        const unsigned int bhi = bhi64 > 0xFFFFFFFFull ? 0xFFFFFFFFu : (unsigned int)bhi64;
        const unsigned int gtau = wtau < bhi ? wtau : bhi;  // the bin's entries: blo <= value < gtau, and not zero (an absent element)
        const int hk = lvl == 1 ? pick_of(hb) : -1;
        if (hk >= 0) {
            const unsigned long long *keys = c.R->picked(c.rr, hk);
            const int m = pk->cnt[hk];
#pragma unroll 1
            for (int i = c.tid; i < m; i += NT) {
                const unsigned long long key = keys[i];
                const unsigned int eb = (unsigned int)(key >> 32);
                if (eb >= blo && eb < gtau) A->cand[satom_add(&A->ncand, 1)] = key;
            }
        } else for_list4(c, [&](const unsigned int (&ebs)[4], int pos0, float *) {
            bool any = false;
#pragma unroll
            for (int u = 0; u < 4; u++) any |= ebs[u] != 0u && ebs[u] >= blo && ebs[u] < gtau;
            if (!__any_sync(0xffffffffu, any)) return;  // one bin of 2048: most warps pass most elements by
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const unsigned int eb = ebs[u];
                if (eb != 0u && eb >= blo && eb < gtau) {
                    const int pos = satom_add(&A->ncand, 1);
                    if (pos < NC) A->cand[pos] = make_key(eb, pos0 + u);
                }
            }
        });
        __syncthreads();
        if (phase < 2 && !try_resume) FSTAMP(12 + 3 * phase);
        const int nb = A->ncand;
        const bool crowded = nb > NC;
        // what lies above the bin is consumed without an event either way
        const float s_bin = binade_ok ? (float)((double)(qy.m0 + qb) * (double)fpow2(j - 23)) : w.s;
        const long long pos_bin = w.pos + ((counting || !binade_ok) ? (long long)cb : 0);
        if (crowded && lvl < 3) {
            w.s = s_bin; w.pos = pos_bin;
            w.tau = bhi < w.tau ? bhi : w.tau;
            lo = blo; shift = (lvl == 1) ? BIN_SHIFT2 : 0; lvl++;
            c.status |= MOLLA_ROW_SLOW_PATH;
            continue;
        }
        if (crowded) {
            // one value, more copies than the buffer holds: add them one at a time (thread 0), then
            // find which copy, in token order, the event fell on
            c.status |= MOLLA_ROW_SLOW_PATH;
            const float pv = __uint_as_float(blo);
            if (c.tid == 0) {
                float s = s_bin;
                long long pos = pos_bin;
                int ev = EV_NONE, at = -1;
#pragma unroll 1
                for (int i = 0; i < nb; i++) {
                    s = __fadd_rn(s, pv);
                    pos++;
                    if (s >= x_ge) ev = EV_CUT;
                    else if (x_gt < s) ev = EV_DRAW;
                    else if (counting && pos >= nstop) ev = EV_LIMIT;
                    if (ev != EV_NONE) { at = i; break; }
                }
                A->b_event = ev; A->b_s = s; A->b_pos = pos; A->b_aux = at;
            }
            __syncthreads();
            const int ev = A->b_event, at = A->b_aux;
            w.s = A->b_s; w.pos = A->b_pos;
            if (ev != EV_NONE) {
                w.event = ev; w.idx = list_nth_equal(c, blo, at); w.p = pv; w.tie = 1;
                return;
            }
            w.tau = blo;
            continue;
        }
        sort_head(c, nb);
        walk_sorted(c, nb, s_bin, pos_bin, x_ge, x_gt, counting, nstop);
        if (phase < 2 && !try_resume) FSTAMP(13 + 3 * phase);
        w.s = A->b_s; w.pos = A->b_pos; w.tau = blo;
        const int ev = A->b_event;
        if (ev != EV_NONE) {
            w.event = ev; w.idx = A->b_idx; w.p = A->b_p; w.tie = A->b_aux;
            __syncthreads();
            return;
        }
        if (phase > 8) c.status |= MOLLA_ROW_SLOW_PATH;
    }
    w.event = EV_DEGENERATE;
    c.status |= MOLLA_ROW_DEGENERATE;
}

// A row that sorts nothing, once tile_walk has written the items of its probabilities: the walk to their
// sum leaves the sum before every stretch, so the draw (sample.mojo:580-590) is a search among those and
// then inside one stretch. Returns false where the general way has to be gone. Bound: latency, of one
// round of loads, the careful chunks' additions, and two more rounds for the values of one item.
__device__ __noinline__ bool tail_pure(CtxF &c) {
    const RowsArgs &R = *c.R;
    WalkShared *W = reinterpret_cast<WalkShared *>(c.A->tile);
    static_assert(sizeof(WalkShared) <= sizeof(AuxF::tile), "the walk fits the tiles' space");
    AuxF *A = c.A;
    const RowHead *head = R.head(c.rr);
    WalkLoads<NT> wl;
    wl.load(R, c.rr);
    const int nitem = head->nitem;
    const float Z = head->Z;
    c.pl = head->plan;
    c.cfg = c.pl.c;
    c.list = R.elist + (size_t)c.rr * R.ntile * TILE;
    c.kmask = R.kmask + (size_t)c.rr * R.ntile * 32;
    const unsigned long long seed = R.a.seed ? R.a.seed[c.cfg.q] : 0ull, drawn = R.a.drawn ? R.a.drawn[c.cfg.q] : 0ull;
    if (nitem > H_ITEMS) return false;
    const unsigned int nrec = wl.order(W, R.ntile, nitem);
    if (nrec > (unsigned int)H_REC) return false;
    FSTAMP(17);
    if (c.warp == 0) {
        float z = 0.0f;
        const bool fine = walk_records(W, R.care(c.rr), c.list, (int)nrec, z);
        if (c.lane == 0) { A->b_s = z; A->b_event = fine ? 1 : 0; A->evt_thread = 0x7fffffff; }
    }
    __syncthreads();
    if (!A->b_event) return false;
    const float sum = A->b_s, target = __fmul_rn(draw01(seed, drawn), sum);
    // the first stretch (runs, then a careful chunk) behind which the sum exceeds the target
#pragma unroll 1
    for (int q = c.tid; q <= (int)nrec; q += NT)
        if (target < __uint_as_float(W->sbs[q + 1])) { atomicMin(&A->evt_thread, q); break; }
    __syncthreads();
    const int q = A->evt_thread;
    FSTAMP(18);
    if (c.warp != 0) return true;
    if (q == 0x7fffffff) {   // the walk fell off the end: the reference returns the last token of the vocabulary
        if (c.lane == 0) finish_row(R.a, c.r, c.cfg, c.status, R.a.V - 1, Z, sum, target, 0.0f);
        return true;
    }
    unsigned int sb = W->sbs[q];
    // 32 items at a time, the records among them counted as order() did: the q-th record's item is the
    // first of the stretch, and the draw falls on a run of the stretch or on the careful chunk at its end
    int seen = 0, item = -1;
    bool in = q == 0;
#pragma unroll 1
    for (int i0 = 0; i0 < nitem && item < 0; i0 += 32) {
        const int i = i0 + c.lane;
        bool rec = false;
        unsigned int ka = 0u;
        if (i < nitem) {
            const Item it = W->items[i];
            rec = it.kind() != K_RUN;
            ka = it.ka;
            if (!rec && !parity_free(it.ka)) rec = true;
            else if (!rec && i > 0) { const Item p = W->items[i - 1]; rec = p.kind() == K_RUN && p.jb() != it.jb(); }
        }
        const unsigned int m = __ballot_sync(0xffffffffu, rec);
        int from = 0;
        if (!in) {
            const int n = __popc(m);
            if (seen + n < q) { seen += n; continue; }
            unsigned int w = m;
#pragma unroll 1
            for (int k = seen + 1; k < q; k++) w &= w - 1u;
            from = __ffs((int)w);      // behind the record before the stretch (which sbs[q] includes)
            in = true;
        }
        const unsigned int later = from < 32 ? m & (0xffffffffu << from) : 0u;
        const int end = later ? __ffs((int)later) - 1 : 32;
        const unsigned int inc = warp_incl_scan(c.lane >= from && c.lane < end ? ka : 0u, c.lane);
        const unsigned int hit = __ballot_sync(0xffffffffu, i < nitem && c.lane >= from && c.lane < end && target < __uint_as_float(sb + inc));
        const int l = hit ? __ffs((int)hit) - 1 : end;
        if (hit) { item = i0 + l; sb += __shfl_sync(0xffffffffu, inc - ka, l); }
        else {
            sb += __shfl_sync(0xffffffffu, inc, 31);
            if (end < 32) item = i0 + end;
        }
    }
    int tile = -1, at = 0;
    if (item >= 0) {
        const Item it = W->items[item];
        const float *v = c.list + (size_t)it.tile() * TILE + it.off();
        int n = it.cnt(), e0 = 0;
        float s = __uint_as_float(sb);
        if (n > 32 && it.kind() == K_RUN) {   // it stays in the sum's binade: each lane adds up the units of its share
            const int per = (n + 31) >> 5, b0 = min(n, c.lane * per), b1 = min(n, b0 + per);
            const unsigned int base = sb & 0x7f800000u;
            float s0 = __uint_as_float(base), s1 = __uint_as_float(base + 1u);
#pragma unroll 8
            for (int e = b0; e < b1; e++) { s0 = __fadd_rn(s0, v[e]); s1 = __fadd_rn(s1, v[e]); }
            const Units k = units_scan(Units{__float_as_uint(s0) - base, __float_as_uint(s1) - base - 1u}, c.lane, 0);
            const unsigned int to = sb + ((sb & 1u) ? k.odd : k.even);
            const unsigned int hit = __ballot_sync(0xffffffffu, target < __uint_as_float(to));
            const int l = hit ? __ffs((int)hit) - 1 : 31;
            if (l > 0) s = __uint_as_float(__shfl_sync(0xffffffffu, to, l - 1));
            e0 = min(n, l * per); n = min(n, e0 + per) - e0;
        }
        int first = -1;
#pragma unroll 1
        for (int g0 = 0; g0 < n && first < 0; g0 += 32) {
            const float mine = g0 + c.lane < n ? v[e0 + g0 + c.lane] : 0.0f;
#pragma unroll 8
            for (int e = 0; e < 32; e++) {
                s = __fadd_rn(s, __shfl_sync(0xffffffffu, mine, e));
                if (first < 0 && g0 + e < n && target < s) first = g0 + e;
            }
        }
        if (first >= 0) { tile = it.tile(); at = it.off() + e0 + first; }
    }
    FSTAMP(10);
    if (c.lane == 0) finish_row(R.a, c.r, c.cfg, c.status, tile < 0 ? R.a.V - 1 : token_of(c, tile, at), Z, sum, target, 0.0f);
    return true;
}

__device__ void tail_row(const RowsArgs &R, int rr) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CtxF c;
    c.tid = threadIdx.x; c.lane = c.tid & 31; c.warp = c.tid >> 5; c.status = 0;
    c.A = reinterpret_cast<AuxF *>(smem_raw);
    c.R = &R;
    AuxF *A = c.A;
    IN_SHARED(A);
    c.rr = rr; c.r = R.r0 + rr;
    const RowHead *head = R.head(rr);
    const int state = head->state;
    FSTAMP(0);
    if (state == ST_PURE) {
        if (tail_pure(c)) return;
        __syncthreads();
    }
    // what the row will look up, in one round of loads: its tiles' entries and items; behind a head that row_head has
    // sorted, the candidates, the walk's ties, the gathered bins and the first binade's table too
    static_assert(MAX_TILES <= 2 * NT && sizeof(AuxF::ties) / 16 <= NT && sizeof(AuxF::u.h) >= NBINS * sizeof(unsigned long long), "a load or two a thread");
    const BatchArgs &a = R.a;
    const int ntile = R.ntile, nhead = state == ST_HEAD ? head->ncand : 0;
    unsigned long long *gcand = R.cand(rr);
    {
        TileOut o[2];
        uint4 vt = make_uint4(0u, 0u, 0u, 0u), vp = vt, x[NBINS / 2 / NT];
        unsigned long long k = 0ull, k0 = 0ull, k1 = 0ull;
        float pre = 0.0f;
#pragma unroll
        for (int u = 0; u < 2; u++)
            if (c.tid + u * NT < ntile) o[u] = R.to(rr)[c.tid + u * NT];
        if (state == ST_HEAD) {
            if (c.tid < (int)(sizeof(A->ties) / 16)) vt = reinterpret_cast<const uint4 *>(R.ties(rr))[c.tid];
            if (c.tid < (int)(sizeof(WalkPicks) / 16)) vp = reinterpret_cast<const uint4 *>(R.picks(rr))[c.tid];
#pragma unroll
            for (int i = 0; i < NBINS / 2 / NT; i++) x[i] = reinterpret_cast<const uint4 *>(R.table(rr, 0))[c.tid + i * NT];
            k = gcand[c.tid]; k0 = c.tid > 0 ? gcand[c.tid - 1] : 0ull; k1 = gcand[c.tid + 1]; pre = R.pre(rr)[c.tid];
        }
        c.pl = head->plan;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int t = c.tid + u * NT;
            if (t < ntile) { A->tcnt[t] = o[u].cnt; A->tni[t] = o[u].nitem; A->tio[t] = o[u].ioff; }
        }
        if (state == ST_HEAD) {
            if (c.tid < (int)(sizeof(A->ties) / 16)) reinterpret_cast<uint4 *>(A->ties)[c.tid] = vt;
            if (c.tid < (int)(sizeof(WalkPicks) / 16)) reinterpret_cast<uint4 *>(&A->picks)[c.tid] = vp;
#pragma unroll
            for (int i = 0; i < NBINS / 2 / NT; i++) reinterpret_cast<uint4 *>(&A->u.h)[c.tid + i * NT] = x[i];
            auto store = [&](int i, unsigned long long key, unsigned long long before, unsigned long long behind, float sum) {
                const unsigned int p = (unsigned int)(key >> 32);
                const bool eq = (i > 0 && (unsigned int)(before >> 32) == p) || (i + 1 < nhead && (unsigned int)(behind >> 32) == p);
                A->pre[i] = sum;
                A->hidx[i] = (unsigned int)key_idx(key) | (eq ? 0x80000000u : 0u);
            };
            if (c.tid < nhead) store(c.tid, k, k0, k1, pre);
#pragma unroll 1
            for (int i = c.tid + NT; i < nhead; i += NT) store(i, gcand[i], gcand[i - 1], i + 1 < nhead ? gcand[i + 1] : 0ull, R.pre(rr)[i]);
        }
    }
    c.cfg = c.pl.c;
    c.list = R.elist + (size_t)c.rr * R.ntile * TILE;
    c.gitems = R.items(rr);
    c.kmask = R.kmask + (size_t)c.rr * R.ntile * 32;
    const RowCfg &g = c.cfg;
    const int imax = c.pl.imax;
    __syncthreads();
    int nc_all = g.pure ? 0 : head->ncand;
    if (nc_all > HEADCAP) {
        __syncthreads();
        if (!(c.pl.flags & F_LIST)) {
#pragma unroll 1
            for (int t = 0; t < ntile; t += SPAN / TILE) tile_again(c, t, min(t + SPAN / TILE, ntile), nullptr, true);
            c.pl.flags |= F_LIST;
        }
        nc_all = narrow_head(c, gcand);
    }
    const bool head_overflow = nc_all > HEADCAP;  // thousands of equal values at the head's edge
    const bool narrow = (c.pl.flags & F_NARROW) != 0;
    if (narrow) c.status |= MOLLA_ROW_SLOW_PATH;

    float dZ = 0.0f, dsum = 0.0f, dtarget = 0.0f, dp = 0.0f;
    int token = -1;
    auto finish = [&]() { FSTAMP(10); if (c.tid == 0) finish_row(a, c.r, g, c.status, token, dZ, dsum, dtarget, dp); };

    // ---- the softmax denominator, exactly as the sequential loop rounds it (sample.mojo:431-434)
    FSTAMP(1);
    const float Z = state != ST_NOTHING ? head->Z : exact_sum(c, false, 0.0f);
    if (state == ST_NOTHING && c.tid == 0) R.head(c.rr)->Z = Z;   // (for jump_status)
    FSTAMP(3);
    dZ = Z;
    const float yZ = __fdiv_rn(1.0f, Z);
    const float u01 = draw01(a.seed ? a.seed[g.q] : 0ull, a.drawn ? a.drawn[g.q] : 0ull);

    // min-p (sample.mojo:508-523) keeps a prefix of the sorted order: the entries whose probability
    // reaches p_max * min_p. Below 2.2e-8 the list no longer holds them all.
    long long n_use = g.n_lim;
    unsigned int minp_pbits = 0u, e_floor = 0u;
    if (g.minp > 0.0f) {
        const float p_top = __fdiv_rn(expf_pinned(__fsub_rn(c.pl.top, c.pl.top)), Z);
        const float floor_p = __fmul_rn(p_top, g.minp);
        minp_pbits = __float_as_uint(floor_p);
        if (!(floor_p >= 2.2e-8f)) { c.status |= MOLLA_ROW_UNSUPPORTED; finish(); return; }
        if (!g.pure) {
            unsigned int lo_b = 0u, hi_b = 0x3F800000u;
#pragma unroll 1
            for (int it = 0; it < 32 && lo_b < hi_b; it++) {
                const unsigned int mid = lo_b + ((hi_b - lo_b) >> 1);
                if (__fdiv_rn(__uint_as_float(mid), Z) >= floor_p) hi_b = mid; else lo_b = mid + 1u;
            }
            e_floor = hi_b;
            int n = 0, tot;
            if (c.pl.flags & F_LIST) {
                for_list4(c, [&](const unsigned int (&eb)[4], int, float *) {
#pragma unroll
                    for (int u = 0; u < 4; u++) n += (eb[u] >= e_floor && eb[u] != 0u) ? 1 : 0;
                });
            } else {
                // the head holds the row's largest, more of them than top-k keeps: a floor below all of it changes nothing
#pragma unroll 1
                for (int i = c.tid; i < nc_all; i += NT) n += (unsigned int)(gcand[i] >> 32) >= e_floor ? 1 : 0;
            }
            (void)block_excl_scan<int>(n, A->wsi, &tot);
            const long long n_ge = tot < 1 ? 1 : tot;  // never empties
            if (n_ge < n_use) n_use = n_ge;
        }
    }

    if (g.pure) {
        // ---- nothing sorted: the draw walks the vocabulary in order (sample.mojo:365-369, 580-594):
        // probabilities p = e / Z (:437-438), what min-p drops becomes zero
#pragma unroll 1
        for (int t = c.warp; t < ntile; t += NWARP) {
            const int n = A->tcnt[t];
            float *src = c.list + (size_t)t * TILE;
            float s = 0.0f;
#pragma unroll 1
            for (int i = c.lane; i < n; i += 32) {
                float p = src[i];
                if (state != ST_PURE) {   // (else tile_walk has done it)
                    p = prob_of(p, Z, yZ);
                    if (__float_as_uint(p) < minp_pbits) p = 0.0f;
                    src[i] = p;
                }
                s += p;
            }
            s = warp_sum(s);
            if (c.lane == 0) A->tsum[t] = s;
        }
        __syncthreads();
        {
            const int t = 2 * c.tid;
            const float s0 = t < ntile ? A->tsum[t] : 0.0f, s1 = t + 1 < ntile ? A->tsum[t + 1] : 0.0f;
            float tot;
            const float ex = block_excl_scan_plus(s0 + s1, A->wsf, &tot);
            __syncthreads();
            if (t < ntile) A->tsum[t] = ex;
            if (t + 1 < ntile) A->tsum[t + 1] = ex + s0;
        }
        __syncthreads();
        float *list = A->tile + (size_t)c.warp * 32 * PITCH;
#pragma unroll 1
        for (int t = c.warp; t < ntile; t += NWARP) {
            const int n = A->tcnt[t];
            const float *src = c.list + (size_t)t * TILE;
#pragma unroll 1
            for (int i = c.lane; i < n; i += 32) list[skew(i)] = src[i];
            __syncwarp();
            const TileChunk ch = tile_chunk(list, n);
            bool care;
            int my_place;
            const int ni = tile_items(list, ch, A->tsum[t], t, c.pl.top, [&](int, int) { return c.gitems + (size_t)t * ITEMS_PER_TILE; }, [](int) { return 255; }, care, my_place);
            if (c.lane == 0) { A->tni[t] = (unsigned short)ni; A->tio[t] = (unsigned int)(t * ITEMS_PER_TILE); }
            __syncwarp();
        }
        __syncthreads();
        const float sum = exact_sum(c, false, 0.0f);
        const float target = __fmul_rn(u01, sum);
        (void)exact_sum(c, true, target);
        dsum = sum; dtarget = target;
        if (A->w_found) {
            if (c.tid == 0) token = token_of(c, A->w_tile, A->w_at);
        } else {
            // the walk fell off the end: the reference returns the last token of the vocabulary,
            // whether or not it could matter to any sum ... or the last one min-p left
            token = a.V - 1;
            if (minp_pbits) {
                int last = -1;
                for_list4(c, [&](const unsigned int (&pb)[4], int pos0, float *) {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (pb[u] >= minp_pbits && pb[u] != 0u) last = max(last, pos0 + u);
                });
                last = __reduce_max_sync(0xffffffffu, last);
                __syncthreads();
                if (c.lane == 0) A->wsi[c.warp] = last;
                __syncthreads();
                for (int w = 0; w < NWARP; w++) last = max(last, A->wsi[w]);
                token = last >= 0 ? token_of(c, last) : imax;
            }
        }
        finish();
        return;
    }

    // ---- sorted order: the head's candidates as probabilities
    const int nc = head_overflow ? 0 : nc_all;
    if (head_overflow) c.status |= MOLLA_ROW_SLOW_PATH;  // no head: the descending walk takes everything from the top
    float head_s;
    long long head_pos;
    if (state == ST_HEAD) {   // row_head has sorted it and added it up
        head_s = head->head_s; head_pos = head->head_pos;
    } else {
    {
#pragma unroll 1
        for (int i = c.tid; i < nc; i += NT) {
            const unsigned long long kk = gcand[i];
            A->cand[i] = ((unsigned long long)__float_as_uint(prob_of(key_val(kk), Z, yZ)) << 32) | (kk & 0xFFFFFFFFull);
        }
    }
    FSTAMP(4);
    sort_head(c, nc);
#pragma unroll 1
    for (int i = c.tid; i < nc; i += NT) {
        const float p = A->pc[i];
        const bool eq = (i > 0 && A->pc[i - 1] == p) || (i + 1 < nc && A->pc[i + 1] == p);
        A->hidx[i] = (unsigned int)key_idx(A->cand[i]) | (eq ? 0x80000000u : 0u);
    }
    __syncthreads();
#ifdef MOLLA_SAMPLE_TESTING
    if (a.topk_out) {
#pragma unroll 1
        for (int i = c.tid; i < a.topk_cap; i += NT)
            a.topk_out[(long long)c.r * a.topk_cap + i] = (i < nc && (long long)i < n_use) ? (int)(A->hidx[i] & 0x7fffffffu) : -1;
    }
#endif
    const bool typ_on = g.typ < 1.0f;
    FSTAMP(5);
    if (c.warp == 0) {
        const HeadEnd e = head_end(HeadRule{g.n_lim, g.P, g.open_row, g.topp_on, g.typ < 1.0f}, a.V, A->pc, A->pre, nc, nc, n_use, narrow, head_overflow, u01);
        if (c.lane == 0) {
            A->b_s = e.s; A->b_pos = e.pos; A->b_event = EV_NONE; A->b_idx = -1; A->b_p = 0.0f; A->b_aux = (int)e.tie;
            if (typ_on) A->ncand = narrow ? -1 : e.cut;  // the typical-p filter takes over from here
            if (e.at >= 0) {
                A->b_event = EV_DRAW; A->b_idx = (int)(A->hidx[e.at] & 0x7fffffffu); A->b_p = A->pc[e.at];
                A->b_sum = e.sum; A->b_target = e.target;
            }
        }
    }
    __syncthreads();
    FSTAMP(6);
    c.status |= (unsigned int)A->b_aux;
    head_s = A->b_s;
    head_pos = A->b_pos;
    if (typ_on) {
        const int m = A->ncand;
        __syncthreads();
        if (m <= 0 || m > HEADC) {
            c.status |= MOLLA_ROW_UNSUPPORTED;  // what the earlier filters left reaches past the head, or is wider than the filter's scratch
        } else {
            typical_head(c, m, g.typ, u01);
            token = A->b_idx; dp = A->b_p; dsum = A->b_sum; dtarget = A->b_target;
            c.status |= (unsigned int)A->b_aux;
        }
        finish();
        return;
    }
    if (A->b_event == EV_DRAW) {
        token = A->b_idx; dp = A->b_p; dsum = A->b_sum; dtarget = A->b_target;
        finish();
        return;
    }
    }

    // ---- past the head: the cut walk, then the draw walk, over the probabilities
    // (sample.mojo:437-438); what the head took is consumed
    const unsigned int tau_bits = head_overflow ? 0xffffffffu : c.pl.tau_bits;
    c.tnb = 0; c.tj0 = 0; c.npick = state == ST_HEAD ? A->picks.n : 0; c.first_table = state == ST_HEAD;
    if (state == ST_HEAD && head_s > 0.0f && fexpo(head_s) >= -30 && fexpo(head_s) < 0) { c.tj0 = fexpo(head_s); c.tnb = min(WALK_BINADES, -c.tj0); }
    if (state != ST_HEAD) for_list4(c, [&](const unsigned int (&eb)[4], int, float *src) {
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (eb[u]) src[u] = eb[u] >= tau_bits ? 0.0f : prob_of(__uint_as_float(eb[u]), Z, yZ);
    });
    __syncthreads();
    FSTAMP(7);
    const bool limited = n_use < (long long)a.V;
    FWalk w;
    FResume resume;
    resume.valid = 0;
    int cut_event = EV_NONE, cut_idx = -1;
    float cut_p = 0.0f, sum = 0.0f, target = 0.0f;
    bool settled = false;    // the token is known, or the row is degenerate
    bool resolved = false;
#pragma unroll 1
    for (int leg = 0; leg < 2; leg++) {   // (one call site for both walks)
        w.s = head_s; w.pos = head_pos; w.tau = 0xFFFFFFFFu;
        w.event = EV_NONE; w.idx = -1; w.p = 0; w.tie = 0;
        const bool cut_round = leg == 0;
        descend_list(c, w, (cut_round && g.topp_on) ? g.P : 3.4e38f, cut_round ? 3.4e38f : target,
                     (cut_round && limited) ? n_use : -1, resume, !cut_round);
        FSTAMP(8 + leg);
        if (!cut_round) {
            if (w.event == EV_DRAW) {
                token = token_of(c, w.idx); dp = w.p; resolved = true;
                if (w.tie) c.status |= MOLLA_ROW_CHOSEN_TIE;
            } else if (w.event == EV_DEGENERATE) {
                resolved = true;
            }
            break;
        }
        cut_event = w.event; cut_idx = w.idx; cut_p = w.p;
        if (cut_event == EV_DEGENERATE) { settled = true; break; }
        if (cut_event == EV_CUT && w.tie) c.status |= MOLLA_ROW_TOPP_TIE;
        if (cut_event == EV_LIMIT && w.tie) c.status |= MOLLA_ROW_TOPK_TIE;
        sum = w.s;
        target = __fmul_rn(u01, sum);
        dsum = sum; dtarget = target;
        // is the drawn element in the head? (the first prefix sum above the target)
        __syncthreads();
        if (c.tid == 0) A->evt_thread = 0x7fffffff;
        __syncthreads();
#pragma unroll 1
        for (int i = c.tid; i < nc; i += NT)
            if (target < A->pre[i]) { atomicMin(&A->evt_thread, i); break; }
        __syncthreads();
        if (A->evt_thread != 0x7fffffff) {
            const int at = A->evt_thread;
            token = (int)(A->hidx[at] & 0x7fffffffu);
            dp = __fsub_rn(A->pre[at], at > 0 ? A->pre[at - 1] : 0.0f);
            if (A->hidx[at] & 0x80000000u) c.status |= MOLLA_ROW_CHOSEN_TIE;
            settled = true;
            break;
        }
        if (!(target < sum)) break;
    }
    if (!settled && !resolved) {
        // the walk falls off the end: the last kept candidate (sample.mojo:591-594)
        if (cut_event == EV_CUT || cut_event == EV_LIMIT) {
            token = token_of(c, cut_idx); dp = cut_p;
        } else {
            // everything listed was kept: its smallest value, highest id last
            unsigned long long best = ~0ull;
            for_list4(c, [&](const unsigned int (&pb)[4], int pos0, float *) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (pb[u]) { const unsigned long long kk = make_key(pb[u], pos0 + u); best = kk < best ? kk : best; }
            });
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                best = ob < best ? ob : best;
            }
            __syncthreads();
            if (c.lane == 0) A->wsu[c.warp] = best;
            __syncthreads();
            for (int v = 0; v < NWARP; v++) best = A->wsu[v] < best ? A->wsu[v] : best;
            token = (best != ~0ull) ? token_of(c, key_idx(best)) : imax;
        }
    }
    finish();
}

// A row that find_jumps has marked: is a guess of its sum's binade wrong? Every marked group's guesses are
// made here as they would be made from that prefix, and held against the sum before them (in double precision,
// added without a subtraction). Pure rows add up twice, exponentials and then probabilities. Bound: latency of code
// that runs once. What comes before is row_plan's estimate but for the tiles that the block and the group
// begin in, so a group takes one or two stretches of logits, evaluated by the whole block; each lane's range is
// added up by four threads. (With whole spans, and a thread for 32 logits or a range, a group took 20 to 45 us:
// row_tail of 160 mixed rows of 2000 31 us where this takes 14, of 256 rows of 151936 76 where this takes 49.)
struct JumpWork { double sum[4][NWARP]; float csum[32]; int jl[32]; int flags[32]; };
static_assert(sizeof(JumpWork) <= ITEM_CAP * sizeof(Item), "the work on a jump uses the items' space");
__device__ __noinline__ void jump_status(const RowsArgs &R, int rr) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AuxF *A = reinterpret_cast<AuxF *>(smem_raw);
    JumpWork &W = *reinterpret_cast<JumpWork *>(A->items);
    const RowHead *head = R.head(rr);
    const RowPlan pl = head->plan;
    const RowCfg &cfg = pl.c;
    const float T = cfg.T, Z = head->Z, f = fminf(1.44269504f / T, 1.0e30f);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = R.r0 + rr, L = R.oL;
    const TilePlan *tp = R.tp + (size_t)rr * R.ntile;
    float minp = 0.0f;   // (nobody's but a pure row's probabilities)
    if (cfg.pure && cfg.minp > 0.0f) minp = __fmul_rn(__fdiv_rn(expf_pinned(__fsub_rn(pl.top, pl.top)), Z), cfg.minp);
    auto prob = [&](float e) -> float {
        const float p = __fdiv_rn(e, Z);
        return p < minp ? 0.0f : p;
    };
    const int npass = cfg.pure ? 2 : 1, nsum = minp > 0.0f ? 4 : 2;
    bool slow = false;
#pragma unroll 1
    for (int q = 0; q < 128 && !slow; q++) {
        const unsigned int left_q = head->hits[q >> 5] >> (q & 31);
        if (!left_q) { q |= 31; continue; }
        q += __ffs((int)left_q) - 1;
        const int blk0 = (q >> 4) * R.oVc, e = min(R.a.V, blk0 + R.oVc), ga = blk0 + (q & 15) * 32 * L, gb = min(e, ga + 32 * L);
        const int t0 = ga / TILE, tb = blk0 / TILE;
        const bool split = tb < t0 && blk0 % TILE != 0;   // the block begins inside a tile before the group's
        double sum[4] = {0.0, 0.0, 0.0, 0.0};   // before the block, in the block before the group; of the probabilities
        if (tid == 0) {
            sum[0] = (double)tp[tb].est;
            if (tb < t0) sum[1] = (double)tp[t0].est - (double)tp[tb + (split ? 1 : 0)].est;
        }
        // the stretches [c0, c1): the block's first tile; where min-p takes something away, everything that it leaves; the group
        const int stop = minp > 0.0f ? t0 * TILE : (split ? (tb + 1) * TILE : 0), step = minp > 0.0f ? SPAN : TILE;
        int c0 = minp > 0.0f ? 0 : tb * TILE;
#pragma unroll 1
        for (bool last = false; !last;) {
            last = c0 >= stop;
            if (last) c0 = t0 * TILE;
            const int c1 = last ? gb : min(c0 + step, stop);
            bool want = last || (split && tb >= c0 / TILE && tb < (c1 + TILE - 1) / TILE);
            for (int t = c0 / TILE; t * TILE < c1 && !want; t++)
                want = ex2_approx((R.ts[(size_t)rr * R.ntile + t].tmax - pl.xmax) * f) >= 0.99f * minp * Z;
            if (want) {
                __syncthreads();
                if (warp < SPAN / TILE && warp * TILE < c1 - c0) span_fetch(R.a, cfg.lrow, c0, A->tile);
                span_ready(R.a, cfg, r, c0, A->tile, reinterpret_cast<SpanScratch *>(A->tile + SPAN_THREADS * PITCH), tid < SPAN_THREADS);
                __syncthreads();
#pragma unroll 1
                for (int i = tid; i < c1 - c0; i += NT) {
                    float &x = A->tile[(i >> 5) * PITCH + (i & 31)];
                    const float ev = x > -INFINITY ? expf_pinned_nonpos(__fsub_rn(T == 1.0f ? x : div_slow(x, T), pl.top)) : 0.0f;
                    x = ev;
                    if (c0 + i < ga) {
                        const bool own = c0 + i >= blk0;
                        if (last || (c0 + i) / TILE == tb) sum[own ? 1 : 0] += (double)ev;
                        if (minp > 0.0f) sum[own ? 3 : 2] += (double)prob(ev);
                    }
                }
            }
            if (!last) c0 = c1;
        }
#pragma unroll 1
        for (int k = 0; k < nsum; k++) {
            double v = k == 0 ? sum[0] : k == 1 ? sum[1] : k == 2 ? sum[2] : sum[3];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) W.sum[k][warp] = v;
        }
        __syncthreads();
#pragma unroll 1
        for (int pass = 0; pass < npass && !slow; pass++) {
            // lane l's range is [i0, i1) of the group, added up four apart, what is left over with the first
            const int n = gb - ga, l = (tid >> 2) & 31, part = tid & 3, i0 = min(n, l * L), i1 = min(n, i0 + L), n4 = (i1 - i0) & ~3;
            auto val = [&](int i) { const int at = ga - c0 + i; const float v = A->tile[(at >> 5) * PITCH + (at & 31)]; return pass ? prob(v) : v; };
            if (tid < 128) {
                float c = 0.0f;
#pragma unroll 1
                for (int i = i0 + part; i < i1; i += i < i0 + n4 ? 4 : 1)
                    if (i < i0 + n4 || part == 0) c = __fadd_rn(c, val(i));
                c = __fadd_rn(c, __shfl_xor_sync(0xffffffffu, c, 1));
                c = __fadd_rn(c, __shfl_xor_sync(0xffffffffu, c, 2));
                if (part == 0) W.csum[l] = c;
            }
            __syncthreads();
            double s0 = 0.0, s1 = 0.0;
            if (warp == 0) {
                double base = 0.0, before = 0.0;
                const int k = pass && minp > 0.0f ? 2 : 0;
#pragma unroll 1
                for (int w = 0; w < NWARP; w++) { base += W.sum[k][w]; before += W.sum[k + 1][w]; }
                if (pass && !(minp > 0.0f)) { base /= (double)Z; before /= (double)Z; }
                const float csum = W.csum[lane];
                const double inc = warp_incl_scan((double)csum, lane), own = __shfl_sync(0xffffffffu, inc, 31);
                double ex = __shfl_up_sync(0xffffffffu, inc, 1);
                if (lane == 0) ex = 0.0;
                const double left = (before + own) - own;   // what the subtraction leaves of `before`
                const double sst = base + (left + (inc - (double)csum));
                const float lo = (float)(sst * (1.0 - 1.0 / 4096.0)), hi = (float)((sst + (double)csum) * (1.0 + 1.0 / 4096.0));
                const int jl = fexpo(lo), j2 = fexpo(hi);
                const bool guessed = lo > 0.0f && csum != 0.0f && j2 <= jl + 1 && jl >= -100 && j2 <= 100;
                W.jl[lane] = jl;
                W.flags[lane] = !guessed ? 0 : (j2 == jl + 1 ? 3 : 1);   // bit 0: there is a guess; bit 1: it spans two binades
                s0 = base + before + ex;
                s1 = s0 + (double)csum;
            }
            __syncthreads();
            if (tid < 128) {   // would the range go by itself in the guessed binades, and does it add anything?
                const int jl = W.jl[l];
                const bool guessed = W.flags[l] != 0, two = W.flags[l] == 3;
                bool bad = false, some = false;
                if (guessed) {
                    const float C1 = __fmul_rn(1.5f, fpow2(jl)), C2 = __fmul_rn(1.5f, fpow2(jl + 1));
#pragma unroll 1
                    for (int i = i0 + part; i < i1; i += 4) {
                        const float v = val(i);
                        const float k1 = __fsub_rn(__fadd_rn(v, C1), C1), k2 = __fsub_rn(__fadd_rn(v, C2), C2);
                        bad |= fabsf(__fsub_rn(v, k1)) == fpow2(jl - 24) || v >= fpow2(jl - 1) || (two && fabsf(__fsub_rn(v, k2)) == fpow2(jl - 23));
                        some |= k1 != 0.0f || (two && k2 != 0.0f);
                    }
                }
                const unsigned int four = 0xfu << (lane & ~3), bm = __ballot_sync(0xffffffffu, bad), sm = __ballot_sync(0xffffffffu, some);
                if (part == 0 && ((bm & four) || !(sm & four))) W.flags[l] = 0;
            }
            __syncthreads();
            bool wrong = false;
            if (warp == 0 && W.flags[lane]) {
                const int jl = W.jl[lane], js = fexpo((float)s0);
                const bool held = W.flags[lane] == 3 ? (js == jl || js == jl + 1) && s1 < (double)fpow2(jl + 2) : js == jl && s1 < (double)fpow2(jl + 1);
                wrong = !held;
            }
            slow = __syncthreads_or(wrong) != 0;
        }
    }
    if (slow && tid == 0) R.a.row_status[r] |= MOLLA_ROW_SLOW_PATH;
}

__global__ void __launch_bounds__(NT, 1) row_tail_kernel(const __grid_constant__ RowsArgs R) {
    if (!R.late_next) pdl_next();
    pdl_wait();
    if (R.late_next) pdl_next();   // (everything before this call's kernels is done by now)
    const int n = R.queue[0];
#pragma unroll 1
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const int rr = R.queue[1 + q];
        if (R.head(rr)->state != ST_DONE) tail_row(R, rr);
        __syncthreads();
        if (R.head(rr)->plan.flags & F_JUMP) {
            // (with the window that the row was sampled with: the token goes into it afterwards)
            jump_status(R, rr);
            __syncthreads();
            if (threadIdx.x == 0) { const int r = R.r0 + rr; took_row(R.a, r, R.head(rr)->plan.c, R.a.tokens[r]); }
        }
    }
}

// ---- host side --------------------------------------------------------------------------------
// The widest layout of one row over thread blocks that F_NARROW speaks of: blocks of at most 38400
// logits, 1, 2, 4 or 8 of them; more than the row needs where the batch leaves the chip idle.
void narrow_layout(int V, int B, int sms, int &oG, int &oVc, int &oL) {
    oG = 0; oVc = 0; oL = 0;
    for (int G = 1; G <= 8; G *= 2) {
        const int Vc = ((((V + G - 1) / G) + 3) / 4) * 4;
        int L = (Vc + NT - 1) / NT;
        if ((L & 1) == 0) L += 1;
        if (L > 75) continue;
        if (oG == 0 || ((long long)B * G * 9 <= (long long)sms * 8 && L >= 9)) { oG = G; oVc = Vc; oL = L; }
    }
}

constexpr long long IN_FLIGHT = 1ll << 27;   // logits whose intermediate results the workspace holds at a time

long long most_in_flight(int V) {
    const long long per = (long long)((V + TILE - 1) / TILE) * TILE;
    return IN_FLIGHT / per > 1 ? IN_FLIGHT / per : 1;
}
int rows_in_flight(int B, int V) {   // a batch that does not fit goes in equal parts
    const long long most = most_in_flight(V), parts = (B + most - 1) / most;
    return (int)((B + parts - 1) / parts);
}
size_t al(size_t n) { return (n + 255) & ~(size_t)255; }

// Lays the rows' intermediate results over the workspace; returns the bytes they take.
size_t lay_out(RowsArgs &A, char *ws, int rows, int V) {
    const size_t nt = (size_t)((V + TILE - 1) / TILE), n = (size_t)rows * nt;
    size_t o = 0;
    auto take = [&](size_t bytes) { char *p = ws + o; o += al(bytes); return p; };
    A.elist = (float *)take(n * TILE * sizeof(float));
    A.gmax = (float *)take(n * 32 * sizeof(float));
    A.kmask = (unsigned int *)take(n * 32 * sizeof(unsigned int));
    A.ts = (TileStat *)take(n * sizeof(TileStat));
    A.tp = (TilePlan *)take(n * sizeof(TilePlan));
    const size_t items = nt * ITEMS_PER_TILE > (size_t)H_ITEMS ? nt * ITEMS_PER_TILE : (size_t)H_ITEMS;
    A.box_stride = (long long)al(sizeof(RowHead) + ((nt + 1) & ~(size_t)1) * sizeof(TileOut) + HEADCAP * (sizeof(unsigned long long) + sizeof(float)) +
                                 CARE_PLACES * 32 * sizeof(float) + items * sizeof(Item));
    A.box = (char *)take((size_t)rows * (size_t)A.box_stride);
    A.walk = take((size_t)rows * WALK_BYTES);
    A.queue = (int *)take((size_t)(rows + 1) * sizeof(int));
    return o;
}

template <class K>
cudaError_t launch(K kernel, unsigned int blocks, unsigned int threads, size_t smem, cudaStream_t st, const RowsArgs &A) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.gridDim = dim3(blocks); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    // every kernel waits for the one before it by itself: its blocks are on the SMs by then
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, A);
}

}  // namespace

size_t molla_rows_workspace_bytes(int B, int V) {
    RowsArgs A;
    const long long most = most_in_flight(V);
    return lay_out(A, nullptr, (int)(B < 1 ? 1 : (B < most ? B : most)), V);
}

int molla_rows_launch(const BatchArgs &a, void *d_workspace, cudaStream_t st, char *err, size_t errlen, float **spare) {
    static bool ready[64] = {};
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && (dev >= 64 || !ready[dev])) {
        e = cudaFuncSetAttribute(tile_stats_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SpanShared));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(tile_exp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SpanShared));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(row_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AuxF));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(tile_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WalkTileShared));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(row_head_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(HeadShared));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(row_head_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(HeadShared));
        if (e == cudaSuccess && dev < 64) ready[dev] = true;
    }
    RowsArgs A;
    A.a = a;
    A.a.Vg = a.V; A.a.col0 = 0; A.a.mode = 0;
    A.ntile = (a.V + TILE - 1) / TILE;
    A.nspan = (a.V + SPAN - 1) / SPAN;
    // of V logits in no order, n reach the value that this share of the lanes' maxima reaches
    const bool far = a.V > HEADCAP && a.V <= FAR_MOST_V;
    auto lanes_for = [&](double n) { return far ? (int)ceil((a.V + 31) / 32 * (1.0 - pow(1.0 - n / a.V, 32.0))) : 0; };
    A.need_far = lanes_for(FAR_HEAD);
    A.need_topk = lanes_for(FAR_TOPK);
    narrow_layout(a.V, a.layout_B > 0 ? a.layout_B : a.B, sms, A.oG, A.oVc, A.oL);
    const int rows = rows_in_flight(a.B, a.V);
    lay_out(A, (char *)d_workspace, rows, a.V);
    // (the lanes' maxima are done with when row_tail begins; 128 bytes a tile of the rows in flight)
    if (spare) *spare = a.B <= 8 * rows ? A.gmax : nullptr;
    for (A.r0 = 0; A.r0 < a.B && e == cudaSuccess; A.r0 += rows) {
        A.late_next = spare && *spare && A.r0 + rows >= a.B;
        A.rows = a.B - A.r0 < rows ? a.B - A.r0 : rows;
        const unsigned int spans = (unsigned int)A.rows * (unsigned int)A.nspan;
        e = launch(tile_stats_kernel, spans, SPAN_THREADS, sizeof(SpanShared), st, A);
        if (e == cudaSuccess) e = launch(row_plan_kernel, (unsigned int)A.rows, NT, 0, st, A);
        if (e == cudaSuccess) e = launch(tile_exp_kernel, spans, SPAN_THREADS, sizeof(SpanShared), st, A);
        if (e == cudaSuccess) e = launch(A.rows > 3 * sms ? row_head_kernel<4> : row_head_kernel<3>, (unsigned int)A.rows, HT, sizeof(HeadShared), st, A);
        if (e == cudaSuccess) e = launch(tile_walk_kernel, spans < 4u * (unsigned int)sms ? spans : 4u * (unsigned int)sms, SPAN_THREADS, sizeof(WalkTileShared), st, A);
        if (e == cudaSuccess) e = launch(tile_pick_kernel, spans < 4u * (unsigned int)sms ? spans : 4u * (unsigned int)sms, SPAN_THREADS, 0, st, A);
        if (e == cudaSuccess) e = launch(row_tail_kernel, (unsigned int)(A.rows < sms ? A.rows : sms), NT, sizeof(AuxF), st, A);
    }
    if (e != cudaSuccess) {
        snprintf(err, errlen, "kernel launch failed: %s", cudaGetErrorString(e));
        return MOLLA_ERR_CUDA;
    }
    return MOLLA_OK;
}
