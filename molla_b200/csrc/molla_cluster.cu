// The row kernel of the ordinary entry points: one logit row per thread-block cluster.
//
// A row of up to 8 x 38400 logits is split into contiguous column ranges, one per thread block
// of the cluster, and every block keeps its range in shared memory from the moment the bulk
// copies (TMA without a tensor map, never multicast) land until the row's token is known. HBM
// sees every logit once and no pass after the first touches global memory: bias and penalties
// are written into the resident range, the maximum is taken from it, the exponentials replace
// the logits in place (what cannot matter to any sum becomes zero, which adds nothing to a
// sequential fp32 sum), and the exact softmax denominator, the sorted head and the walks past
// it all read shared memory. The range's position is the token id, so nothing carries indices.
//
// What the blocks of a cluster have to tell each other (the range maxima, a lower bound of the
// running sum before each range, the threads' maxima for the head threshold, the estimated
// range sums, the exact running sum handed from range to range, the head's candidates, the
// bin tables of a walk) goes through distributed shared memory between cluster barriers. All
// blocks of a cluster take the same branches: every decision is made from values all of them
// hold.
//
// The device functions this kernel shares with the streaming kernel (the exact sum, the bin
// search, the sorted walk, typical-p) come from molla_exact.cuh.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stddef.h>
#include <stdio.h>

#include "molla_exact.cuh"
#include "molla_cluster.h"

namespace cg = cooperative_groups;

namespace {

constexpr int CL_MAX_G = 8;                  // thread blocks per cluster at most (the portable limit)
constexpr int CL_LMAX = 75;                  // logits per thread at most (odd: conflict-free strides)
constexpr int CL_CAPF = NT * CL_LMAX;        // logits per thread block at most: 38400 (150 KB)
constexpr int CL_PIECE = 4096;               // floats per bulk copy
constexpr int CL_HEADC = HEADCAP;             // candidates of the sorted head at most (the buffers of a gathered bin hold as many)
constexpr int CL_HEAD_NEED = HEAD_MOST;
constexpr int TIE_CAP = 64;                   // rounding ties a walk resolves by parity; more send it the slow way
constexpr int TBINS = NT;                    // bins of the threads' maxima by distance below the row's maximum
constexpr float TRES = (float)(NT / 32);     // bins per unit of logit: the bins cover 32 units

// Profiling stamps exist in the testing build only (per row 32 slots of clock readings and counts).
#ifdef MOLLA_SAMPLE_TESTING
#define CSTAMP(i) do { if (a.prof && leader && c.tid == 0) a.prof[(long long)r * 32 + (i)] = clock64(); } while (0)
#define CPROF_SLOTS(cond, first) ((a.prof && (cond)) ? a.prof + (long long)r * 32 + (first) : nullptr)
#else
#define CSTAMP(i) do { } while (0)
#define CPROF_SLOTS(cond, first) nullptr
#endif

// A piece of a block's range as the exact sum goes through it: chunks (a thread's logits) whose binade is certain,
// a chunk or a warp of them that may lie in either of two, or a chunk to be added value by value.
struct __align__(16) Stretch {
    unsigned int ka, kb;   // pairs of units in binade jb, and in the next one
    unsigned int meta;     // biased exponent of the binade (8 bits; 255: value by value), it may be the next one (1 bit);
                           // what was guessed: the binade (8 bits; 0: nothing), two of them (1); place of the values (8; 255: none)
    unsigned int where;    // first chunk (9 bits), chunks (10 bits)
    __device__ __forceinline__ unsigned int jb() const { return meta & 0xffu; }
    __device__ __forceinline__ unsigned int both() const { return (meta >> 8) & 1u; }
    __device__ __forceinline__ unsigned int guess() const { return (meta >> 9) & 0xffu; }
    __device__ __forceinline__ bool guess_two() const { return (meta >> 17) & 1u; }
    __device__ __forceinline__ int place() const { return (int)((meta >> 18) & 0xffu); }
    __device__ __forceinline__ int first() const { return (int)(where & 511u); }
    __device__ __forceinline__ int chunks() const { return (int)(where >> 9); }
    __device__ __forceinline__ bool run() const { return jb() != 255u && !both(); }
};
constexpr int RECS = 64;                     // stretches of a block that the leader has at hand

// walk_fast's own.
constexpr int FAST_RECS = 160;
// units of all plain stretches before it, its own; binade of the last of those (8 bits), guess (8), two binades guessed (1), place (8), whether it has units (1)
struct __align__(16) FastRec { unsigned int k, ka, kb, meta; };

struct __align__(16) AuxC {
    union {
        struct {
            Stretch items[NWARP * 33];        // of this block's range, in order
            Stretch recs[CL_MAX_G][RECS];     // leader: of every block, runs across warps as one
            FastRec fast[FAST_RECS];          // leader: see walk_fast
            float after[FAST_RECS];           // the sum behind each of them,
            unsigned short org[FAST_RECS];    // and which stretch it is: block (3 bits), number (9)
        } p1;
        struct {
            unsigned int hq[NBINS];
            unsigned int hqh[NBINS];
            unsigned int hc[NBINS];
        } h;
    } u;
    unsigned long long cand[NC];   // first the hash of the patched tokens, then the head / a bin's candidates
    float pc[NC];
    float pre[CL_HEADC];
    unsigned int hidx[CL_HEADC];
    double wsd[2 * (NWARP + 1)];
    unsigned long long wsu[NWARP + 1];
    float wsf[NWARP + 1];
    int wsi[NWARP + 1];
    int ncand, evt_thread, specbin, hit_bin;
    unsigned long long hit_qbefore, hit_cbefore, tot_q, tot_c;
    float b_s; int b_event; int b_idx; float b_p; long long b_pos; int b_aux;
    float b_sum; float b_target;
    uint64_t mbar;
    unsigned int thist[TBINS];           // the threads' maxima by distance below the block's maximum
    // what the blocks of the cluster write into each other (slot = the writer's rank)
    float x1_max[CL_MAX_G]; int x1_idx[CL_MAX_G]; int x1_eq[CL_MAX_G]; unsigned int x1_status[CL_MAX_G];
    float x2_total[CL_MAX_G];
    double x3_tot[CL_MAX_G]; int x3_n[CL_MAX_G];
    int x4_n[CL_MAX_G]; unsigned long long x5_key[CL_MAX_G];
    int nitem, nrec[CL_MAX_G], nfast;            // stretches of this block; leader: of every block; of walk_fast, or -1
    float first_s[CL_MAX_G];                     // leader: the sum before every block
    float ch_s; int ch_at, ch_slow;              // the exact sum as the leader found it
    // elements of a walk that would round on a tie: their keys, bins, the mass before them
    long long rx[8];          // words fetched from the leader for the whole block
    int ngath, ngath_over;   // a bin's entries collected by this block; blocks whose own buffer overflowed (leader's)
    int ntie[2]; unsigned long long tkey[TIE_CAP]; int tbin[TIE_CAP]; unsigned char tord[TIE_CAP]; unsigned int tpq_lo[TIE_CAP], tpq_hi[TIE_CAP]; unsigned long long tpqm[TIE_CAP], tabove[TIE_CAP], tc[TIE_CAP];
    unsigned int tbits[NBINS / 32];
    int r_kind; int r_idx; float r_s; long long r_pos; unsigned int r_status;  // the leader's word after the head
};

struct CtxC {
    int tid, lane, warp;
    AuxC *A;
    unsigned int status;
};
// (What is called out of line makes its own: a reference to the kernel's would put that on the stack, and every loop with an
// atomic in it would load the thread's number from there again. The walks past the head took a tenth longer so.)
__device__ __forceinline__ CtxC ctx_of(AuxC *A) {
    CtxC c;
    c.tid = threadIdx.x; c.lane = c.tid & 31; c.warp = c.tid >> 5; c.status = 0;
    c.A = A;
    return c;
}

struct ClWalk {
    float s; long long pos; unsigned int tau;
    int event; int idx; float p; int tie;
};

struct ClGeo {          // where this thread block stands
    int G, rank, c0, nloc, L;
};

// The exact sequential fp32 sum of the cluster's row (values `bits`, zero = absent), in vocabulary
// order. Every thread turns its chunk of the range into units of the binade (or two) in which the estimated sum
// before it says the sum will be, every warp its chunks into stretches, every block its warps' into as few as may be,
// which go to the leader with the values of the chunks that may have to be added one by one. One warp of the leader
// goes through them: a stretch inside a binade is one addition, the chunk in which the sum leaves a binade is added
// value by value. A guess that the exact sum shows to be wrong is made good for from the values.
struct ClSum { float s; int slow; };

// (every lane of the warp calls these and gets the same answer)
__device__ __noinline__ unsigned int add_chunk(const float *v, int n, unsigned int sb) {
    const int lane = threadIdx.x & 31;
    float s = __uint_as_float(sb);
#pragma unroll 1
    for (int i = 0; i < n; i += 32) {
        const float mine = i + lane < n ? v[i + lane] : 0.0f;
#pragma unroll 8
        for (int e = 0; e < 32; e++) s = __fadd_rn(s, __shfl_sync(0xffffffffu, mine, e));
    }
    return __float_as_uint(s);
}

// MOLLA_ROW_SLOW_PATH tells a caller that a guess of the sum's binade went wrong: whether that is said of a chunk
// whose guess (binade jb, or that and the next one) did not hold. Not where nothing was added, and not where the
// chunk held a rounding tie or a value of a quarter of the binade: such chunks never went by their guess.
__device__ __noinline__ bool guess_counts(const float *v, int n, unsigned int jb, bool two) {
    const int j = (int)jb - 127;
    const float C1 = __fmul_rn(1.5f, fpow2(j)), C2 = __fmul_rn(1.5f, fpow2(j + 1));
    bool bad = false, some = false;
    for (int i = 0; i < n; i++) {
        const float x = v[i], k1 = __fsub_rn(__fadd_rn(x, C1), C1), k2 = __fsub_rn(__fadd_rn(x, C2), C2);
        bad |= fabsf(__fsub_rn(x, k1)) == fpow2(j - 24) || x >= fpow2(j - 1) || (two && fabsf(__fsub_rn(x, k2)) == fpow2(j - 23));
        some |= k1 != 0.0f || (two && k2 != 0.0f);
    }
    return some && !bad;
}
__device__ __forceinline__ bool guess_held(unsigned int jb, bool two, unsigned int before, unsigned int after) {
    const unsigned int e = before >> 23, f = after >> 23;
    return jb == 0u || ((e == jb || (two && e == jb + 1u)) && f <= jb + (two ? 1u : 0u));
}

// One thread's units: its values added to the smallest even and the smallest odd pattern of the binade with biased exponent e.
template <class V>
__device__ __forceinline__ Units chunk_units(V lst, int i0, int i1, unsigned int e) {
    const unsigned int base = e << 23;
    float s0 = __uint_as_float(base), s1 = __uint_as_float(base + 1u);
#pragma unroll 4
    for (int i = i0; i < i1; i++) { const float v = lst(i); s0 = __fadd_rn(s0, v); s1 = __fadd_rn(s1, v); }
    return Units{__float_as_uint(s0) - base, __float_as_uint(s1) - base - 1u};
}

struct ChunksSum { unsigned int sb; bool slow; };
// Chunks [first, first + n) of a block's values, whatever was guessed about them.
__device__ __noinline__ ChunksSum add_chunks(const float *vals, int nloc, int L, int first, int n, unsigned int sb, unsigned int jb, bool two) {
    const int lane = threadIdx.x & 31;
    ChunksSum r{sb, false};
#pragma unroll 1
    for (int c0 = first; c0 < first + n; c0 += 32) {
        const int m = min(32, first + n - c0), i0 = min(nloc, (c0 + lane) * L), i1 = lane < m ? min(nloc, i0 + L) : i0;
        bool wrong = false;
        int at = 0;
#pragma unroll 1
        while (at < m) {
            const unsigned int e = r.sb >> 23;
            const Units d = units_scan(lane < at ? Units{0u, 0u} : chunk_units([&](int i) { return vals[i]; }, i0, i1, e), lane, 0);
            const unsigned int to = r.sb + ((r.sb & 1u) ? d.odd : d.even);
            unsigned int from = __shfl_up_sync(0xffffffffu, to, 1);
            if (lane == 0) from = r.sb;
            const unsigned int stop = __ballot_sync(0xffffffffu, lane >= at && lane < m && (to >> 23) != e);
            const int f = stop ? __ffs((int)stop) - 1 : m;
            if (lane >= at && lane < f) wrong |= !guess_held(jb, two, from, to);
            if (f > at) r.sb = __shfl_sync(0xffffffffu, to, f - 1);
            at = f;
            if (at < m) {
                const int o = min(nloc, (c0 + at) * L);
                const unsigned int q = add_chunk(vals + o, min(nloc, o + L) - o, r.sb);
                if (lane == at) wrong |= !guess_held(jb, two, r.sb, q);
                r.sb = q;
                at++;
            }
        }
        if (__any_sync(0xffffffffu, wrong)) r.slow |= __any_sync(0xffffffffu, wrong && guess_counts(vals + i0, i1 - i0, jb, two)) != 0;
    }
    return r;
}

// Where the values of chunks to be added one by one wait for the leader's walk, `pitch` floats each: over pc, pre and
// hidx, half of the places for the leader's own range, in which most binades are crossed.
__device__ __forceinline__ int care_pitch(int L) { return (L + 11) / 12 * 12; }   // (whole steps of add_place)
__device__ __forceinline__ void care_places(int L, int G, int rank, int &first, int &n) {
    static_assert(offsetof(AuxC, pre) == offsetof(AuxC, pc) + sizeof(AuxC::pc) && offsetof(AuxC, hidx) == offsetof(AuxC, pre) + sizeof(AuxC::pre), "one area");
    static_assert(offsetof(AuxC, pc) % 16 == 0, "read four at a time");
    const int all = min(255, (int)((sizeof(AuxC::pc) + sizeof(AuxC::pre) + sizeof(AuxC::hidx)) / sizeof(float)) / care_pitch(L));
    const int own = G == 1 ? all : all / 2, others = G == 1 ? 0 : (all - own) / (G - 1);
    first = rank == 0 ? 0 : own + (rank - 1) * others;
    n = rank == 0 ? own : others;
}

// A place's values added to s, twelve at a time with the next twelve's loads ahead. (Addresses as numbers: through
// pointers the loads were generic ones, with 64-bit arithmetic around them.)
__device__ __forceinline__ float4 lds4(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float add_place(const AuxC *A, int place, int pitch4, float s) {
    uint32_t at = smem_u32(A->pc) + (uint32_t)(place * pitch4) * 16u;
    const uint32_t last = at + (uint32_t)(pitch4 - 3) * 16u;
    float4 x[3] = {lds4(at), lds4(at + 16u), lds4(at + 32u)};
#pragma unroll 2
    for (; at <= last; at += 48u) {
        const uint32_t n = min(at + 48u, last);
        const float4 y[3] = {lds4(n), lds4(n + 16u), lds4(n + 32u)};
#pragma unroll
        for (int u = 0; u < 3; u++) { s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, x[u].x), x[u].y), x[u].z), x[u].w); x[u] = y[u]; }
    }
    return s;
}

// The usual row: no guess is wrong. The leader's first warp first strings the stretches of all blocks together, 32 at a
// time: those that are plain additions become part of what lies before the next that is not, and only
// these (ten or twenty: mostly the chunks in which the sum leaves a binade) are gone through one by one. (Every
// instruction of that loop is one of a lone warp's, eight cycles or so: with the plain ones in it, it took 14 thousand.)
// Returns false, and nothing else, where something does not hold.
__device__ __noinline__ bool walk_fast(AuxC *A, ClGeo g, int Vc, int V, const unsigned int *bits, float &sum) {
    IN_SHARED(A);
    cg::cluster_group cl = cg::this_cluster();
    const CtxC c = ctx_of(A);
    const int lane = c.lane, pitch4 = care_pitch(g.L) / 4;
    const unsigned int lt = (1u << lane) - 1u;
    const int cnt = lane < g.G ? A->nrec[lane] : 0, incl = warp_incl_scan(cnt, lane), total = __shfl_sync(0xffffffffu, incl, 31);
    if (lane == 0) A->nfast = -1;
    if (__any_sync(0xffffffffu, cnt > RECS)) return false;
    FastRec *out = A->u.p1.fast;
    int ncare = 0;
    unsigned int k = 0u, carry = 0u;   // of the record before this batch: its binade, 0 where it was not a run
#pragma unroll 1
    for (int b = 0; b < total; b += 32) {
        const int idx = b + lane;
        int h = 0, at = idx;
#pragma unroll
        for (int o = 0; o < CL_MAX_G - 1; o++) {
            const int end = __shfl_sync(0xffffffffu, incl, o);
            if (o < g.G - 1 && idx >= end) { h = o + 1; at = idx - end; }
        }
        const bool have = idx < total;
        Stretch it;
        it.ka = it.kb = it.where = 0u; it.meta = 255u;
        if (have) it = A->u.p1.recs[h][at];
        const unsigned int rj = it.run() ? it.jb() : 0u;
        unsigned int pj = __shfl_up_sync(0xffffffffu, rj, 1);
        if (lane == 0) pj = carry;
        carry = __shfl_sync(0xffffffffu, rj, 31);
        const bool care = have && (!it.run() || !parity_free(it.ka) || (pj != 0u && pj != rj));
        const unsigned int inc = warp_incl_scan(have && !care ? it.ka : 0u, lane), cm = __ballot_sync(0xffffffffu, care);
        const int i = ncare + __popc(cm & lt);
        if (care && i < FAST_RECS - 1) {
            FastRec r;
            r.k = k + inc; r.ka = it.ka; r.kb = it.kb;
            r.meta = pj | (it.guess() << 8) | (it.guess_two() ? 1u << 16 : 0u) | ((unsigned int)(it.chunks() > 1 ? 255 : it.place()) << 17) | (it.jb() != 255u ? 1u << 25 : 0u);
            out[i] = r;
            A->u.p1.org[i] = (unsigned short)(h << 9 | at);
        }
        ncare += __popc(cm);
        k += __shfl_sync(0xffffffffu, inc, 31);
        if (b + 32 >= total) carry = __shfl_sync(0xffffffffu, rj, (total - 1) & 31);
    }
    if (ncare >= FAST_RECS - 1) return false;
    if (lane == 0) { FastRec r; r.k = k; r.ka = r.kb = 0u; r.meta = carry; out[ncare] = r; }
    __syncwarp();
    unsigned int sb = 0u, kdone = 0u;
    FastRec nx = out[0];
#pragma unroll 1
    for (int q = 0; ; q++) {
        const FastRec r = nx;
        nx = out[min(q + 1, ncare)];
        const unsigned int to = sb + (r.k - kdone), jr = r.meta & 0xffu, e = to >> 23;
        if (jr != 0u && ((sb >> 23) != jr || e != jr)) return false;   // (also where the runs add nothing)
        kdone = r.k;
        sb = to;
        if (q == ncare) break;
        const unsigned int jb = (r.meta >> 8) & 0xffu, both = (r.meta >> 16) & 1u, d = e - jb, td = to + units(d ? r.kb : r.ka, to);
        if (((r.meta >> 25) & 1u) && d <= both && (td >> 23) == e) sb = td;
        else {
            const int place = (int)((r.meta >> 17) & 0xffu);
            if (place != 255) sb = __float_as_uint(add_place(A, place, pitch4, __uint_as_float(to)));
            else {   // several chunks, or one that found no place: out of its block's memory
                const int o = A->u.p1.org[q], h = o >> 9, nloc = max(0, min(Vc, V - h * Vc));
                const Stretch it = A->u.p1.recs[h][o & 511];
                const float *vals = reinterpret_cast<const float *>(h == 0 ? bits : cl.map_shared_rank(const_cast<unsigned int *>(bits), h));
                if (it.chunks() > 1) {
                    const ChunksSum s = add_chunks(vals, nloc, g.L, it.first(), it.chunks(), to, it.guess(), it.guess_two());
                    if (s.slow) return false;
                    sb = s.sb;
                } else {
                    const int i0 = min(nloc, it.first() * g.L);
                    sb = add_chunk(vals + i0, min(nloc, i0 + g.L) - i0, to);
                }
            }
            // (where a binade was guessed: the guess held?)
            if (jb != 0u && !(d <= both && (sb >> 23) <= jb + both)) return false;
        }
        if (lane == 0) A->u.p1.after[q] = __uint_as_float(sb);
    }
    if (lane == 0) A->nfast = ncare;
    sum = __uint_as_float(sb);
    return true;
}

// The leader's first warp, all lanes alike, whatever was guessed: through the stretches from number i0 of block h0 on, the sum before them sb. With
// `locate`, ends with the stretch behind which the sum exceeds `target`: its block, place and the sum before it.
struct Walked { unsigned int sb; bool slow; int h, first, chunks; };
__device__ __noinline__ Walked walk_stretches(AuxC *A, ClGeo g, int Vc, int V, const unsigned int *bits, int h0, int i0, unsigned int sb, bool locate, float target) {
    IN_SHARED(A);
    cg::cluster_group cl = cg::this_cluster();
    const CtxC c = ctx_of(A);
    Walked w{sb, false, -1, 0, 0};
    const int pitch4 = care_pitch(g.L) / 4;
#pragma unroll 1
    for (int h = h0; h < g.G; h++) {
        const int nrec = A->nrec[h];
        const bool far = nrec > RECS;   // (too many: where the block has left them)
        const int n = far ? cl.map_shared_rank(A, h)->nitem : nrec;
        const Stretch *list = far ? cl.map_shared_rank(A, h)->u.p1.items : A->u.p1.recs[h];
        if (!locate && c.lane == 0) A->first_s[h] = __uint_as_float(w.sb);
        const int from = h == h0 ? i0 : 0;
        if (from >= n) continue;
        Stretch nx = list[from];
#pragma unroll 1
        for (int i = from; i < n; i++) {
            const Stretch it = nx;
            nx = list[min(i + 1, n - 1)];
            const unsigned int before = w.sb, e = before >> 23, d = e - it.jb(), to = before + units(d ? it.kb : it.ka, before);
            if (d <= it.both() && (to >> 23) == e) w.sb = to;
            else {
                const int nloc = max(0, min(Vc, V - h * Vc)), o = min(nloc, it.first() * g.L), len = min(nloc, o + g.L) - o;
                const float *vals = reinterpret_cast<const float *>(h == 0 ? bits : cl.map_shared_rank(const_cast<unsigned int *>(bits), h));
                if (it.chunks() > 1) {
                    const ChunksSum q = add_chunks(vals, nloc, g.L, it.first(), it.chunks(), before, it.guess(), it.guess_two());
                    w.sb = q.sb; w.slow |= q.slow;
                } else {
                    if (it.place() == 255) w.sb = add_chunk(vals + o, len, before);
                    else {
                        const float s = add_place(A, it.place(), pitch4, __uint_as_float(before));
                        w.sb = __float_as_uint(s);
                    }
                    if (!guess_held(it.guess(), it.guess_two(), before, w.sb)) w.slow |= guess_counts(vals + o, len, it.guess(), it.guess_two());
                }
            }
            if (locate && target < __uint_as_float(w.sb)) {
                w.sb = before; w.h = h; w.first = it.first(); w.chunks = it.chunks();
                return w;
            }
        }
    }
    return w;
}

__device__ __noinline__ ClSum cluster_exact_sum(AuxC *A, ClGeo g, int Vc, int V, const unsigned int *bits, long long *stamps = nullptr) {
    IN_SHARED(A);
    cg::cluster_group cl = cg::this_cluster();
    const CtxC c = ctx_of(A);
    IN_SHARED(bits);
    AuxC *lead = cl.map_shared_rank(A, 0);
    ValBits vals{bits};
    __syncthreads();
    const float csum = p1_csum(vals, g.nloc, g.L, c.tid);
    double tot;
    const double ex = block_excl_scan<double>((double)csum, A->wsd, &tot);
    if (c.tid < g.G) cl.map_shared_rank(A, c.tid)->x3_tot[g.rank] = tot;
    cl.sync();
    double sbase = 0.0;
    for (int h = 0; h < g.rank; h++) sbase += A->x3_tot[h];
    if (stamps && c.tid == 0) stamps[0] = clock64();
    const double sst = sbase + ex;
    // the binade of the sum before and behind this chunk; 2^-12 covers the rounding of the true one
    const float EPS = 1.0f / 4096.0f;
    const float lo = (float)(sst * (1.0 - (double)EPS)), hi = (float)((sst + (double)csum) * (1.0 + (double)EPS));
    const int i0 = min(g.nloc, c.tid * g.L), i1 = min(g.nloc, (c.tid + 1) * g.L), lane = c.lane;
    const int jl = fexpo(lo), jh = fexpo(hi);
    const bool nonempty = i1 > i0 && csum != 0.0f;
    const bool usable = nonempty && lo > 0.0f && jh <= jl + 1 && jl >= -100 && jh <= 100, two = usable && jh == jl + 1;
    const unsigned int jb = (unsigned int)(jl + 127);
    Units da{0u, 0u}, db{0u, 0u};
    bool over = false;   // outgrows a binade by itself
    if (usable) {
        da = chunk_units(vals, i0, i1, jb);
        over = ((jb << 23) + 1u + da.odd) >> 23 != jb;
    }
    if (__any_sync(0xffffffffu, two) && two) {
        db = chunk_units(vals, i0, i1, jb + 1u);
        over |= (((jb + 1u) << 23) + 1u + db.odd) >> 23 != jb + 1u;
    }
    // A run that adds nothing is none, unless the sum may still be in the binade below (each of the additions before took 2^-24
    // of it at most), where it might add something: then it is a stretch of no units, by which the binade is checked.
    const unsigned int um = __ballot_sync(0xffffffffu, usable && (da.even | da.odd) == 0u && fexpo(lo * (1.0f - (float)(g.c0 + i1) * (1.0f / 16777216.0f))) < jl);
    const bool step = nonempty && (!usable || over);
    const unsigned int ne = __ballot_sync(0xffffffffu, nonempty), lt = (1u << lane) - 1u, below = ne & lt;
    const int prev = below ? 31 - __clz((int)below) : lane;
    const int pj = __shfl_sync(0xffffffffu, jl, prev);
    const bool prev_alone = ((__ballot_sync(0xffffffffu, step || two) >> prev) & 1u) != 0u;
    const int j0 = __shfl_sync(0xffffffffu, jl, max(__ffs((int)ne) - 1, 0));
    // (chunks that all may lie in the same two binades are one stretch: a sum that stays near a power of two for long)
    const bool merged = __popc(ne) >= 8 && __all_sync(0xffffffffu, !nonempty || (two && !over && jl == j0));
    const bool care = !merged && (step || two || (nonempty && below && !prev_alone && pj != jl));
    const unsigned int cm = __ballot_sync(0xffffffffu, care), cb = cm & lt;
    const int lastc = cb ? 31 - __clz((int)cb) : -1, last = cm ? 31 - __clz((int)cm) : -1;
    const Units ra = units_scan(care || !usable ? Units{0u, 0u} : da, lane, care ? lane : lastc + 1);
    const unsigned int kp = pair_of(ra.even, ra.odd);
    unsigned int kr = __shfl_up_sync(0xffffffffu, kp, 1);
    if (lane == 0) kr = 0u;
    auto behind = [&](int l) { return l < 0 ? 0xffffffffu : ~((2u << l) - 1u); };   // the lanes past l
    const unsigned int runm = __ballot_sync(0xffffffffu, care && (kr != 0u || (um & lt & behind(lastc)) != 0u));
    const unsigned int ktail = last == 31 || merged ? 0u : __shfl_sync(0xffffffffu, kp, 31);
    const bool tail = ktail != 0u || (!merged && (um & behind(last)) != 0u);
    const int n = merged ? 1 : __popc(cm) + __popc(runm) + (tail ? 1 : 0);
    if (lane == 0) A->wsi[c.warp] = n | (__popc(cm) << 16);
    Units rb{0u, 0u};
    if (merged) rb = units_scan(db, lane, 0);
    auto first_in = [&](int from) { const unsigned int m = ne & ~(from < 0 ? 0u : (from == 31 ? 0xffffffffu : ((2u << from) - 1u))); return m ? __ffs((int)m) - 1 : 31; };
    const int fj = __shfl_sync(0xffffffffu, jl, first_in(lastc)), tj = __shfl_sync(0xffffffffu, jl, first_in(last));
    __syncthreads();
    int at = 0;
    for (int w = 0; w < c.warp; w++) at += A->wsi[w];
    int place0, places;
    care_places(g.L, g.G, g.rank, place0, places);
    const int care0 = at >> 16;
    at &= 0xffff;
    if (c.tid == NT - 1) A->nitem = at + n;
    Stretch *out = A->u.p1.items + at;
    const unsigned int w0 = (unsigned int)c.warp * 32u;
    auto stretch = [&](unsigned int ka, unsigned int kb, unsigned int match, bool both, int guess, bool guess_two, int place, unsigned int first, unsigned int chunks) {
        Stretch it;
        it.ka = ka; it.kb = kb;
        it.meta = match | (both ? 1u << 8 : 0u) | ((unsigned int)(guess + 127) << 9) | (guess_two ? 1u << 17 : 0u) | ((unsigned int)place << 18);
        it.where = (w0 + first) | (chunks << 9);
        return it;
    };
    int place = 255;
    if (care) {
        int i = __popc(cb) + __popc(runm & lt);
        const int nth = care0 + __popc(cb);
        place = nth < places ? place0 + nth : 255;
        if ((runm >> lane) & 1u) out[i++] = stretch(kr, 0u, (unsigned int)(fj + 127), false, fj, false, 255, (unsigned int)(lastc + 1), (unsigned int)(lane - lastc - 1));
        const bool known = usable && !over;
        out[i] = stretch(known ? pair_of(da.even, da.odd) : 0u, known && two ? pair_of(db.even, db.odd) : 0u, known ? jb : 255u, known && two, usable ? jl : -127, two, place,
                         (unsigned int)lane, 1u);
    }
    if (lane == 31 && merged) out[0] = stretch(kp, pair_of(rb.even, rb.odd), (unsigned int)(j0 + 127), true, j0, true, 255, 0u, 32u);
    if (lane == 31 && tail) out[n - 1] = stretch(ktail, 0u, (unsigned int)(tj + 127), false, tj, false, 255, (unsigned int)(last + 1), (unsigned int)(31 - last));
    // the careful chunks' values to the leader, padded with zeros
    const int pitch = care_pitch(g.L);
    for (unsigned int left = __ballot_sync(0xffffffffu, place != 255); left; left &= left - 1u) {
        const int l = __ffs((int)left) - 1, o = __shfl_sync(0xffffffffu, i0, l), len = __shfl_sync(0xffffffffu, i1, l) - o;
        float *to = lead->pc + __shfl_sync(0xffffffffu, place, l) * pitch;
        for (int i = lane; i < pitch; i += 32) to[i] = i < len ? vals(o + i) : 0.0f;
    }
    __syncthreads();
    if (c.warp == 0) {   // the block's stretches to the leader, runs of one binade across warps as one
        const int total = A->nitem;
        int nrec = 0;
        for (int b = 0; b < total; b += 32) {
            const bool have = b + lane < total;
            Stretch it;
            it.ka = it.kb = it.where = 0u; it.meta = 255u;
            if (have) it = A->u.p1.items[b + lane];
            const bool run = it.run(), before = __shfl_up_sync(0xffffffffu, run, 1);
            const unsigned int mj = it.jb(), bj = __shfl_up_sync(0xffffffffu, mj, 1);
            const unsigned int starts = __ballot_sync(0xffffffffu, lane == 0 || !run || !before || bj != mj);
            const int s0 = 31 - __clz((int)(starts & (lt | (1u << lane))));
            const unsigned int w_first = __shfl_sync(0xffffffffu, it.where, s0) & 511u;
            Units u{units(it.ka, 0u), units(it.ka, 1u)};
            if (__any_sync(0xffffffffu, run && !parity_free(it.ka))) u = units_scan(u, lane, s0);
            else {
                const unsigned int inc = warp_incl_scan(run ? u.even : 0u, lane), b0 = __shfl_sync(0xffffffffu, inc, max(s0 - 1, 0));
                u.even = u.odd = inc - (s0 > 0 ? b0 : 0u);
            }
            const bool ends = have && (lane == 31 || ((starts >> (lane + 1)) & 1u) || b + lane + 1 == total);
            const unsigned int em = __ballot_sync(0xffffffffu, ends);
            const int i = nrec + __popc(em & lt);
            if (run) {
                it.ka = pair_of(u.even, u.odd);
                it.where = w_first | (((it.where & 511u) + (it.where >> 9) - w_first) << 9);
            }
            if (ends && i < RECS) lead->u.p1.recs[g.rank][i] = it;
            nrec += __popc(em);
        }
        if (lane == 0) lead->nrec[g.rank] = nrec;
    }
    if (stamps && c.tid == 0) stamps[1] = clock64();
    cl.sync();
    if (g.rank == 0 && c.warp == 0) {
        Walked w{0u, false, -1, 0, 0};
        float sum;
        if (walk_fast(A, g, Vc, V, bits, sum)) w.sb = __float_as_uint(sum);
        else w = walk_stretches(A, g, Vc, V, bits, 0, 0, 0u, false, 0.0f);
        if (lane < g.G) { AuxC *ox = cl.map_shared_rank(A, lane); ox->ch_s = __uint_as_float(w.sb); ox->ch_slow = w.slow ? 1 : 0; }
    }
    cl.sync();
    return ClSum{A->ch_s, A->ch_slow};
}

// The token at which the running sum of the last cluster_exact_sum (`total`) first exceeds `target`, or -1. Its
// stretches and the values they stand for are where it left them.
__device__ __noinline__ int cluster_locate(AuxC *A, ClGeo g, int Vc, int V, const unsigned int *bits, float total, float target) {
    IN_SHARED(A);
    cg::cluster_group cl = cg::this_cluster();
    const CtxC c = ctx_of(A);
    IN_SHARED(bits);
    if (!(target < total)) return -1;   // (the same in every block)
    if (g.rank == 0 && c.warp == 0) {
        // from behind the last careful stretch, or from the last block, that the sum did not exceed the target at (it never falls)
        int h = 0, i = 0;
        float s = 0.0f;
        if (A->nfast >= 0) {
            int n = 0;
            for (int q = c.lane; q < A->nfast; q += 32) if (!(target < A->u.p1.after[q])) n = q + 1;
            n = __reduce_max_sync(0xffffffffu, n);
            if (n > 0) { const int o = A->u.p1.org[n - 1]; h = o >> 9; i = (o & 511) + 1; s = A->u.p1.after[n - 1]; }
        } else {
            for (int k = 0; k < g.G; k++) if (!(target < A->first_s[k])) { h = k; s = A->first_s[k]; }
        }
        const Walked w = walk_stretches(A, g, Vc, V, bits, h, i, __float_as_uint(s), true, target);
        if (c.lane < g.G) {
            AuxC *ox = cl.map_shared_rank(A, c.lane);
            ox->r_kind = w.h; ox->r_idx = w.first | (w.chunks << 16); ox->r_s = __uint_as_float(w.sb);
            ox->ch_at = -1;
        }
    }
    cl.sync();
    if (A->r_kind == g.rank) {   // the block that holds it: every thread the sum before its chunk, the first one past the target looks into it
        const int first = A->r_idx & 0xffff, n = A->r_idx >> 16;
        const unsigned int sb = __float_as_uint(A->r_s), e = sb >> 23;
        const int i0 = min(g.nloc, c.tid * g.L), i1 = min(g.nloc, i0 + g.L);
        ValBits vals{bits};
        const bool mine = c.tid >= first && c.tid < first + n;
        unsigned int before = sb, to = sb;
        if (n > 1) {
            const Units d = units_scan(mine ? chunk_units(vals, i0, i1, e) : Units{0u, 0u}, c.lane, 0);
            __syncthreads();
            if (c.lane == 31) A->wsu[c.warp] = (unsigned long long)d.even | ((unsigned long long)d.odd << 32);
            __syncthreads();
            Units base{0u, 0u};
            for (int w = 0; w < c.warp; w++) base = then(base, Units{(unsigned int)A->wsu[w], (unsigned int)(A->wsu[w] >> 32)});
            const Units all = then(base, d), up{__shfl_up_sync(0xffffffffu, all.even, 1), __shfl_up_sync(0xffffffffu, all.odd, 1)}, mb = c.lane == 0 ? base : up;
            to = sb + ((sb & 1u) ? all.odd : all.even);
            before = sb + ((sb & 1u) ? mb.odd : mb.even);
        }
        if (c.tid == 0) A->evt_thread = 0x7fffffff;
        __syncthreads();
        // (a sum that leaves the binade inside: the guess was wrong, or it is one chunk; then from the first of them on)
        const bool left = n == 1 || __syncthreads_or(mine && (to >> 23) != e) != 0;
        if (left) { if (c.tid == first) { A->evt_thread = first; before = sb; } }
        else if (mine && target < __uint_as_float(to)) atomicMin(&A->evt_thread, c.tid);
        __syncthreads();
        if (A->evt_thread == c.tid) {
            float s = __uint_as_float(before);
            int found = -1;
            for (int i = i0; i < (left ? min(g.nloc, (first + n) * g.L) : i1); i++) {
                s = __fadd_rn(s, vals(i));
                if (target < s) { found = i; break; }
            }
            for (int o = 0; o < g.G; o++) cl.map_shared_rank(A, o)->ch_at = found < 0 ? -1 : g.c0 + found;
        }
    }
    cl.sync();
    return A->ch_at;
}

// Token id of the (nth+1)-th entry, in vocabulary order, whose bits equal `eb` (eb below tau).
__device__ int cluster_nth_equal(cg::cluster_group &cl, CtxC &c, const ClGeo &g, const unsigned int *bits,
                                 unsigned int eb, int nth) {
    AuxC *A = c.A;
    IN_SHARED(A);
    IN_SHARED(bits);
    const int i0 = min(g.nloc, c.tid * g.L), i1 = min(g.nloc, (c.tid + 1) * g.L);
    int cnt = 0;
    for (int i = i0; i < i1; i++) cnt += (bits[i] == eb) ? 1 : 0;
    int tot;
    const int ex = block_excl_scan<int>(cnt, A->wsi, &tot);
    if (c.tid < g.G) cl.map_shared_rank(A, c.tid)->x4_n[g.rank] = tot;
    if (c.tid == 0) A->r_idx = -1;
    cl.sync();
    int base = 0;
    for (int h = 0; h < g.rank; h++) base += A->x4_n[h];
    if (nth >= base + ex && nth < base + ex + cnt) {
        int seen = base + ex;
        for (int i = i0; i < i1; i++) {
            if (bits[i] == eb) {
                if (seen == nth) {
                    for (int o = 0; o < g.G; o++) cl.map_shared_rank(A, o)->r_idx = g.c0 + i;
                    break;
                }
                seen++;
            }
        }
    }
    cl.sync();
    return A->r_idx;
}

// A few words of the leader's memory for the whole block: threads 0..n-1 fetch one each into
// `A->rx` (a load from another block's memory by every thread would queue up there).
template <class F>
__device__ __forceinline__ void fetch_from_leader(CtxC &c, int n, F word) {
    __syncthreads();
    if (c.tid < n) c.A->rx[c.tid] = word(c.tid);
    __syncthreads();
}

// This block's elements below `tau` and from `lo` on into the tables of a walk whose sum lies in binade j: those that add a
// number of units that does not depend on the sum, by bin; a rounding tie to the leader's list, the bin of any
// other to specbin. With `count_all`, their number too. Out of line, with registers of its own: in line the loop's
// share of the kernel's depended on what else was in it (120 rows of 32000 with a top-k of 1024 42 to 51 thousand cycles).
// Every thread's elements four at a time. The common case (an element that simply adds its
// mass to its bin) runs without a branch; elements that need care and rounding ties are rare
// and a warp turns to them only when one of its lanes has met one.
__device__ __noinline__ void walk_tables(AuxC *A, AuxC *lead, const unsigned int *bits, int nloc, int c0, unsigned int tau, unsigned int lo, int shift, int j,
                                         bool binade_ok, bool count_all, bool ties_listed, int ntie_slot) {
    IN_SHARED(A);
    IN_SHARED(bits);
    const float Cm = __fmul_rn(1.5f, fpow2(j)), halfu = fpow2(j - 24), bigthr = fpow2(j - 1);
    const unsigned int cm_bits = __float_as_uint(Cm);
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i0 = threadIdx.x - lane; i0 < nloc; i0 += 4 * NT) {  // (the same trips for all lanes of a warp)
        const int i4 = i0 + lane;
        unsigned int ebs[4];
        bool rare = false;
#pragma unroll
        for (int u = 0; u < 4; u++) ebs[u] = (i4 + u * NT < nloc) ? bits[i4 + u * NT] : 0u;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const unsigned int eb = ebs[u];
            const bool live = eb != 0u && eb < tau && eb >= lo;
            const int bin = (int)((eb - lo) >> shift);
            const float p = __uint_as_float(eb);
            const float tq = __fadd_rn(p, Cm);
            const float q = __fsub_rn(tq, Cm);
            const float rr = __fsub_rn(p, q);
            const bool special = (fabsf(rr) == halfu) || (p >= bigthr);
            // q in units: below bigthr, p + Cm stays in Cm's binade, whose unit is the sum's, so
            // the difference of the two bit patterns is the count (a conversion would issue at
            // a quarter of the rate)
            const unsigned int qu = __float_as_uint(tq) - cm_bits;
            if (live && count_all) sred_add(&A->u.h.hc[bin], 1u);
            const bool plain = live && binade_ok && !special;
            if (plain) sred_add(&A->u.h.hq[bin], qu & MASS_LO_MASK);
            if (plain && (qu >> MASS_SPLIT)) sred_add(&A->u.h.hqh[bin], qu >> MASS_SPLIT);
            rare |= live && binade_ok && special;
        }
        if (__any_sync(0xffffffffu, rare)) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const unsigned int eb = ebs[u];
                if (!(eb != 0u && eb < tau && eb >= lo)) continue;
                const int bin = (int)((eb - lo) >> shift);
                const float p = __uint_as_float(eb);
                const float q = __fsub_rn(__fadd_rn(p, Cm), Cm);
                const bool tie = fabsf(__fsub_rn(p, q)) == halfu;
                if ((p >= bigthr) || (tie && !ties_listed)) { sred_max(&A->specbin, bin); continue; }
                if (tie) {
                    const int pos = atomicAdd(&lead->ntie[ntie_slot], 1);
                    if (pos < TIE_CAP) { lead->tkey[pos] = make_key(eb, c0 + i4 + u * NT); lead->tbin[pos] = bin; }
                }
            }
        }
    }
}


// The descending walk past the sorted head (sample.mojo:492-506 and :580-590) over the cluster's
// row of probabilities. State as in `descend`: exact running sum, elements consumed, and tau:
// everything with probability bits >= tau is consumed. Every phase histograms what remains by
// value bin (each block its range; the tables are added up across the cluster as they are
// read), consumes whole bins up to the first one holding an event, gathers that bin into the
// leader's candidate buffer, and the leader sorts it and adds it element by element.
//
// An element whose addition would be a rounding tie (its value is an odd multiple of half the
// running sum's unit) rounds up or down with the parity of the sum before it. Such elements do
// not stop a phase: they are listed, a second pass adds up what precedes each of them inside
// its own bin, and one thread then resolves them from the top down, each from the exact integer
// sum before it; their contributions go into their bins' masses before the event is searched.
// Where a walk's last phase began. The draw walk adds up the same elements in the same order as
// the cut walk before it, so when its target is not reached before that point it starts there,
// on the bin tables that are still standing (merged, at the leader), and skips the passes that
// built them.
struct ClResume {
    int valid;
    float s; long long pos; unsigned int tau;
    int lvl; unsigned int lo; int shift; int tie_mode; int ntie;
};

__device__ void descend_cluster(cg::cluster_group &cl, CtxC &c, const ClGeo &g, const unsigned int *bits,
                                ClWalk &w, float x_ge, float x_gt, long long nstop, ClResume &rs, bool try_resume,
                                long long *dbg = nullptr) {
    AuxC *A = c.A;
    IN_SHARED(A);
    IN_SHARED(bits);
    AuxC *lead = cl.map_shared_rank(A, 0);
    const bool leader = g.rank == 0;
    const bool counting = nstop >= 0;
    int lvl = 1;
    unsigned int lo = 0u;
    int shift = BIN_SHIFT;
    bool tie_mode = true;
    // (every block holds the same `rs`: its fields are values all blocks computed alike)
    const bool resumed = try_resume && rs.valid && !counting && x_ge >= 3.0e38f && !(x_gt < rs.s);
    if (resumed) {
        w.s = rs.s; w.pos = rs.pos; w.tau = rs.tau;
        lvl = rs.lvl; lo = rs.lo; shift = rs.shift; tie_mode = rs.tie_mode != 0;
    }
    if (c.tid == 0) { A->ntie[0] = 0; A->ntie[1] = 0; }
    for (int phase = 0; phase < 8192; phase++) {
        const bool reuse = resumed && phase == 0;  // this phase's tables stand already
        cl.sync();  // nobody still reads the tables or the leader's results of the phase before
        long long tp0 = clock64();
#define DT(k) do { if (dbg && c.tid == 0) { const long long t_ = clock64(); dbg[k] += t_ - tp0; tp0 = t_; } } while (0)
        if (!reuse) {
            for (int i = c.tid; i < NBINS; i += NT) { A->u.h.hq[i] = 0u; A->u.h.hqh[i] = 0u; A->u.h.hc[i] = 0u; }
            for (int i = c.tid; i < NBINS / 32; i += NT) A->tbits[i] = 0u;
            rs.valid = 1; rs.s = w.s; rs.pos = w.pos; rs.tau = w.tau;
            rs.lvl = lvl; rs.lo = lo; rs.shift = shift; rs.tie_mode = tie_mode ? 1 : 0; rs.ntie = 0;
        }
        if (c.tid == 0) {
            if (!reuse) A->specbin = -1;
            A->ncand = 0; A->ngath = 0; A->ngath_over = 0; A->ntie[(phase + 1) & 1] = 0;  // the other blocks add to this phase's counter already
        }
        __syncthreads();
        const bool have_s = w.s > 0.0f;
        const int j = have_s ? fexpo(w.s) : 0;
        const bool binade_ok = have_s && j >= -100 && j <= 100;
        const float Cm = __fmul_rn(1.5f, fpow2(j)), halfu = fpow2(j - 24), bigthr = fpow2(j - 1);
        const float inv_u = fpow2(23 - j);
        const unsigned int cm_bits = __float_as_uint(Cm);
        const bool ties_listed = tie_mode && lvl == 1 && binade_ok;
        int ntie = rs.ntie;
        if (!reuse) {
        const int ntie_slot = phase & 1;
        walk_tables(A, lead, bits, g.nloc, g.c0, w.tau, lo, shift, j, binade_ok, counting || !binade_ok, ties_listed, ntie_slot);
        cl.sync();
        fetch_from_leader(c, 1, [&](int) { return (long long)lead->ntie[ntie_slot]; });
        ntie = ties_listed ? (int)A->rx[0] : 0;
        rs.ntie = ntie;
        if (dbg && c.tid == 0) { dbg[0] += 1; dbg[1] += ntie; }
        DT(3);
        if (ntie > TIE_CAP) { tie_mode = false; c.status |= MOLLA_ROW_SLOW_PATH; continue; }  // too many: they stop phases instead
        if (ntie > 0) {
            // what precedes each listed element inside its own bin (descending value, then ascending id)
            if (c.tid < ntie) {
                const int b = lead->tbin[c.tid];
                A->tkey[c.tid] = lead->tkey[c.tid]; A->tbin[c.tid] = b; A->tpq_lo[c.tid] = 0u; A->tpq_hi[c.tid] = 0u;
                sred_or(&A->tbits[b >> 5], 1u << (b & 31));
            }
            __syncthreads();
            // the bins that hold a listed element span a short range: a compare against it keeps
            // nearly every element out of the slower path
            int tb_lo = NBINS, tb_hi = -1;
            for (int t = 0; t < ntie; t++) { tb_lo = min(tb_lo, A->tbin[t]); tb_hi = max(tb_hi, A->tbin[t]); }
            const unsigned int tb_span = (unsigned int)(tb_hi - tb_lo);

            const unsigned int wtau2 = w.tau;
            for (int i0 = c.tid - c.lane; i0 < g.nloc; i0 += 4 * NT) {
                const int i4 = i0 + c.lane;
                unsigned int ebs[4];
                bool near = false;
#pragma unroll
                for (int u = 0; u < 4; u++) ebs[u] = (i4 + u * NT < g.nloc) ? bits[i4 + u * NT] : 0u;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned int eb = ebs[u];
                    const int bin = (int)((eb - lo) >> shift);
                    near |= eb != 0u && eb < wtau2 && eb >= lo && (unsigned int)(bin - tb_lo) <= tb_span;
                }
                if (!__any_sync(0xffffffffu, near)) continue;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned int eb = ebs[u];
                    if (eb == 0u || eb >= wtau2 || eb < lo) continue;
                    const int bin = (int)((eb - lo) >> shift);
                    if (!((A->tbits[bin >> 5] >> (bin & 31)) & 1u)) continue;
                    const float p = __uint_as_float(eb);
                    const float tq = __fadd_rn(p, Cm);
                    const float q = __fsub_rn(tq, Cm);
                    const float rr = __fsub_rn(p, q);
                    if (fabsf(rr) == halfu || p >= bigthr) continue;
                    const unsigned int qu = __float_as_uint(tq) - cm_bits;
                    const unsigned long long key = make_key(eb, g.c0 + i4 + u * NT);
                    for (int t = 0; t < ntie; t++)
                        if (A->tbin[t] == bin && key > A->tkey[t] && qu) {  // two halves, as in the bin tables
                            sred_add(&A->tpq_lo[t], qu & MASS_LO_MASK);
                            if (qu >> MASS_SPLIT) sred_add(&A->tpq_hi[t], qu >> MASS_SPLIT);
                        }
                }
            }
            cl.sync();
        }
        }  // (!reuse)
        DT(4);
        // The leader adds the other blocks' tables to its own (whole rows of bins at a time, so that
        // the loads from the other blocks' memory are few and wide), searches the event bin and
        // tells everybody.
        BinQuery qy;
        qy.bin_hi = NBINS; qy.spec_bits = nullptr;
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
        if (!reuse && g.G > 1) {
            // every block adds up its share of the bins over all blocks (few, wide loads from the
            // other blocks' memory, spread over all of them) and puts the sums into the leader's tables
            uint4 *mine = reinterpret_cast<uint4 *>(&A->u.h);
            uint4 *dst = reinterpret_cast<uint4 *>(&lead->u.h);
            constexpr int NV = 3 * NBINS / 4;  // the three tables, four bins at a time
            const int per = (NV + g.G - 1) / g.G;
            const int v_hi = min(NV, (g.rank + 1) * per);
            for (int v0 = g.rank * per + c.tid; v0 < v_hi; v0 += NT) {
                uint4 acc = mine[v0];
                for (int o = 0; o < g.G; o++) {
                    if (o == g.rank) continue;
                    const uint4 x = reinterpret_cast<const uint4 *>(&cl.map_shared_rank(A, o)->u.h)[v0];
                    acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
                }
                dst[v0] = acc;
            }
            if (!leader && c.tid == 0 && A->specbin >= 0) atomicMax(&lead->specbin, A->specbin);
            cl.sync();
        }
        if (leader) {
            if (reuse) {
                if (c.tid < ntie) A->tc[c.tid] = 0ull;
                __syncthreads();
            } else {
                if (c.tid < ntie) {
                    unsigned long long s_ = 0ull;
                    for (int o = 0; o < g.G; o++) {
                        const AuxC *ox = cl.map_shared_rank(A, o);
                        s_ += (unsigned long long)ox->tpq_lo[c.tid] + ((unsigned long long)ox->tpq_hi[c.tid] << MASS_SPLIT);
                    }
                    A->tpqm[c.tid] = s_; A->tc[c.tid] = 0ull;
                }
                __syncthreads();
            }
            qy.specbin = A->specbin;
            find_event_bin_adj(c, qy,
                [&](int b, unsigned long long &q, unsigned long long &n) {
                    q = (unsigned long long)qy.hq[b] + ((unsigned long long)qy.hqh[b] << MASS_SPLIT);
                    n = qy.hc[b];
                },
                [&](unsigned long long (&q)[BPT], unsigned long long eq) -> bool {
                    if (ntie == 0) return false;
                    // the mass before each listed element: the bins above its own (the thread that
                    // owns the bin knows), what precedes it inside the bin (added up over the blocks)
                    unsigned long long run = eq;
#pragma unroll
                    for (int i = 0; i < BPT; i++) {
                        const int b = NBINS - 1 - BPT * c.tid - i;
                        for (int t = 0; t < ntie; t++)
                            if (A->tbin[t] == b) A->tabove[t] = run;
                        run += q[i];
                    }
                    if (c.tid < ntie) {   // the ties' order from the top
                        int rank = 0;
                        for (int t = 0; t < ntie; t++) rank += A->tkey[t] > A->tkey[c.tid] ? 1 : 0;
                        A->tord[rank] = (unsigned char)c.tid;
                    }
                    __syncthreads();
                    if (c.tid == 0) {
                        // from the top down (what lies below an event never matters: the walk stops there)
                        unsigned long long carried = 0ull;
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
                        for (int t = 0; t < ntie; t++)
                            if (A->tbin[t] == b) q[i] += A->tc[t];
                    }
                    return true;
                });
            if (c.tid < g.G && c.tid > 0) {
                AuxC *ox = cl.map_shared_rank(A, c.tid);
                ox->hit_bin = A->hit_bin; ox->hit_qbefore = A->hit_qbefore; ox->hit_cbefore = A->hit_cbefore;
                ox->tot_q = A->tot_q; ox->tot_c = A->tot_c;
            }
        }
        cl.sync();
        DT(5);
        const int hb = A->hit_bin;
        if (hb < 0) {
            // nothing left in this range triggers an event: consume it whole
            if (binade_ok) w.s = (float)((double)(qy.m0 + A->tot_q) * (double)fpow2(j - 23));
            w.pos += (long long)A->tot_c;
            if (lvl == 1) { w.tau = 0; w.event = EV_EXHAUSTED; cl.sync(); return; }
            w.tau = lo; lvl = 1; lo = 0u; shift = BIN_SHIFT;  // back to the coarse bins below this range
            continue;
        }
        const unsigned long long qb = A->hit_qbefore, cb = A->hit_cbefore;
        const unsigned int blo = lo + ((unsigned int)hb << shift);
        const unsigned long long bhi64 = (unsigned long long)lo + ((unsigned long long)(hb + 1) << shift);
        const unsigned int bhi = bhi64 > 0xFFFFFFFFull ? 0xFFFFFFFFu : (unsigned int)bhi64;
        // The bin's entries: every block collects its own (in the space of the candidates' values),
        // reserves room at the leader with one addition to the leader's counter and copies them over.
        unsigned long long *mybuf = reinterpret_cast<unsigned long long *>(A->pc);
        constexpr int MYCAP = NC / 2;
        const unsigned int gtau = w.tau < bhi ? w.tau : bhi;  // the bin's entries: blo <= value < gtau, and not zero (an absent element)
        for (int i0 = c.tid - c.lane; i0 < g.nloc; i0 += 4 * NT) {  // (the same trips for all lanes of a warp)
            const int i4 = i0 + c.lane;
            unsigned int ebs[4];
            bool any = false;
#pragma unroll
            for (int u = 0; u < 4; u++) ebs[u] = (i4 + u * NT < g.nloc) ? bits[i4 + u * NT] : 0u;
#pragma unroll
            for (int u = 0; u < 4; u++) any |= ebs[u] != 0u && ebs[u] >= blo && ebs[u] < gtau;
            if (!__any_sync(0xffffffffu, any)) continue;  // one bin of 2048: most warps pass most elements by
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const unsigned int eb = ebs[u];
                if (eb != 0u && eb >= blo && eb < gtau) {
                    const int pos = satom_add(&A->ngath, 1);
                    if (pos < MYCAP) mybuf[pos] = make_key(eb, g.c0 + i4 + u * NT);
                }
            }
        }
        __syncthreads();
        const int mine = A->ngath;
        if (c.tid == 0) {
            A->evt_thread = atomicAdd(&lead->ncand, mine);  // (a word that is idle here; the leader's `specbin` has to survive for a resumed walk)
            if (mine > MYCAP) atomicAdd(&lead->ngath_over, 1);  // more than this block could hold: the bin is split further
        }
        __syncthreads();
        const int cbase = A->evt_thread;
        if (mine <= MYCAP && cbase + mine <= NC)
            for (int i = c.tid; i < mine; i += NT) lead->cand[cbase + i] = mybuf[i];
        cl.sync();
        fetch_from_leader(c, 2, [&](int i) { return (long long)(i == 0 ? lead->ncand : lead->ngath_over); });
        const int nb = (int)A->rx[0];
        const bool crowded = nb > NC || A->rx[1] > 0;
        DT(6);
        if (dbg && c.tid == 0) dbg[2] = nb;
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
            // one value, more copies than the buffer holds: add them one at a time (the leader's
            // thread 0), then find which copy, in token order, the event fell on
            c.status |= MOLLA_ROW_SLOW_PATH;
            const float pv = __uint_as_float(blo);
            if (g.rank == 0 && c.tid == 0) {
                float s = s_bin;
                long long pos = pos_bin;
                int ev = EV_NONE, at = -1;
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
            cl.sync();
            fetch_from_leader(c, 4, [&](int i) {
                return i == 0 ? (long long)lead->b_event : i == 1 ? (long long)lead->b_aux
                     : i == 2 ? (long long)__float_as_int(lead->b_s) : lead->b_pos; });
            const int ev = (int)A->rx[0], at = (int)A->rx[1];
            w.s = __int_as_float((int)A->rx[2]); w.pos = A->rx[3];
            if (ev != EV_NONE) {
                const int id = cluster_nth_equal(cl, c, g, bits, blo, at);
                w.event = ev; w.idx = id; w.p = pv; w.tie = 1;
                return;
            }
            w.tau = blo;
            continue;
        }
        if (g.rank == 0) {
            sort_cands(c, nb);
            walk_sorted(c, nb, s_bin, pos_bin, x_ge, x_gt, counting, nstop);
        }
        cl.sync();
        DT(7);
        fetch_from_leader(c, 6, [&](int i) {
            return i == 0 ? (long long)lead->b_event : i == 1 ? (long long)lead->b_aux
                 : i == 2 ? (long long)__float_as_int(lead->b_s) : i == 3 ? lead->b_pos
                 : i == 4 ? (long long)lead->b_idx : (long long)__float_as_int(lead->b_p); });
        w.s = __int_as_float((int)A->rx[2]); w.pos = A->rx[3]; w.tau = blo;
        const int ev = (int)A->rx[0];
        if (ev != EV_NONE) {
            w.event = ev; w.idx = (int)A->rx[4]; w.p = __int_as_float((int)A->rx[5]); w.tie = (int)A->rx[1];
            cl.sync();  // the leader's results are read before anyone moves on
            return;
        }
        if (phase > 8) c.status |= MOLLA_ROW_SLOW_PATH;
    }
    w.event = EV_DEGENERATE;
    c.status |= MOLLA_ROW_DEGENERATE;
}

__global__ void __launch_bounds__(NT, 1) sample_rows_cluster_kernel(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    cg::cluster_group cl = cg::this_cluster();
    float *rowbuf = reinterpret_cast<float *>(smem_raw);
    unsigned int *rowbits = reinterpret_cast<unsigned int *>(smem_raw);
    AuxC *A = reinterpret_cast<AuxC *>(smem_raw + (size_t)CL_CAPF * 4);
    CtxC c = ctx_of(A);
    IN_SHARED(A);
    IN_SHARED(rowbuf);
    IN_SHARED(rowbits);
    ClGeo g;
    g.G = a.G; g.rank = (int)cl.block_rank(); g.L = a.L;
    g.c0 = g.rank * a.Vc;
    g.nloc = max(0, min(a.Vc, a.V - g.c0));
    const int r = (int)blockIdx.x / g.G;
    const bool leader = g.rank == 0;
    AuxC *lead = cl.map_shared_rank(A, 0);

    // ---- settings (the same in every block of the cluster)
    const int q = a.slot ? a.slot[r] : r;
    const long long lrow = a.rows ? (long long)a.rows[r] : (long long)r;
    const bool idx_ok = (!a.slot || (q >= 0 && (a.n_slots <= 0 || q < a.n_slots))) &&
                        (!a.rows || (lrow >= 0 && (a.n_logit_rows <= 0 || lrow < a.n_logit_rows)));
    if (!idx_ok) {  // a stale row or slot index: nothing of that row or slot is touched
        if (leader && c.tid == 0) { a.tokens[r] = -1; a.row_status[r] = MOLLA_ROW_INVALID_CONFIG; }
        return;
    }
    const float T = a.temperature ? a.temperature[q] : 0.0f;
    const int k = a.top_k ? a.top_k[q] : 0;
    const float P = a.top_p ? a.top_p[q] : 1.0f;
    const float minp = a.min_p ? a.min_p[q] : 0.0f;
    const float typ = a.typical_p ? a.typical_p[q] : 1.0f;
    const float rp = a.repeat_penalty ? a.repeat_penalty[q] : 1.0f;
    const float fp = a.frequency_penalty ? a.frequency_penalty[q] : 0.0f;
    const float pp = a.presence_penalty ? a.presence_penalty[q] : 0.0f;
    const int ring_n = a.ring ? min(max(a.ring_len[q], 0), a.ring_cap) : 0;
    const bool won = a.ring ? (ring_n > 0) : (a.window_on ? (a.window_on[q] != 0) : true);
    const int h0 = (a.hist && a.hist_off) ? a.hist_off[q] : 0;
    const long long *histp = a.ring ? a.ring + (size_t)q * (size_t)a.ring_cap : (a.hist ? a.hist + h0 : nullptr);
    const int H = a.ring ? min(max(a.ring_filled[q], 0), ring_n) : ((a.hist && a.hist_off) ? (a.hist_off[q + 1] - h0) : 0);
    const int b0 = (a.bias_ids && a.bias_off) ? a.bias_off[q] : 0;
    const int nb = (a.bias_ids && a.bias_off) ? (a.bias_off[q + 1] - b0) : 0;
    // the rules of SamplerConfig.check (sample.mojo:140-154); NaN fails every test
    const bool valid = (T >= 0.0f) && (k >= 0) && (P > 0.0f && P <= 1.0f) && (minp >= 0.0f && minp <= 1.0f) &&
                       (typ > 0.0f && typ <= 1.0f) && (rp > 0.0f) && H >= 0 && nb >= 0;
    const bool greedy = !(T > 0.0f);
    const bool penalizing = won && H > 0 && (rp != 1.0f || fp != 0.0f || pp != 0.0f);
    const int npatch = (penalizing ? H : 0) + nb;
    if (!valid) c.status |= MOLLA_ROW_INVALID_CONFIG;
    // typical-p is done on rows an earlier filter sorted and cut to a set inside the sorted head
    else if (!greedy && typ < 1.0f && !((k > 0 && k < a.V) || P < 1.0f)) c.status |= MOLLA_ROW_UNSUPPORTED;
    if (npatch > PATCH_MAX) c.status |= MOLLA_ROW_UNSUPPORTED;

    float dZ = 0.0f, dsum = 0.0f, dtarget = 0.0f, dp = 0.0f;
    int token = -1;
    // the end of every row: the leader's thread 0 writes the answer and does `_took`
    auto finish = [&]() {
        if (!(leader && c.tid == 0)) return;
#ifdef MOLLA_SAMPLE_TESTING
        if (a.prof) {
            unsigned long long gt;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(gt));
            a.prof[(long long)r * 32 + 11] = (long long)gt; a.prof[(long long)r * 32 + 9] = clock64();
        }
#endif
        if (c.status & (MOLLA_ROW_LOAD_TIMEOUT | MOLLA_ROW_DEGENERATE | MOLLA_ROW_INVALID_CONFIG | MOLLA_ROW_UNSUPPORTED | MOLLA_ROW_EMPTY)) token = -1;
        a.tokens[r] = token;
        a.row_status[r] = c.status;
        if (a.ring && token >= 0) {  // `_took` (sample.mojo:361-363): observe, then one more draw used
            if (ring_n > 0) {        // `observe` (:246-258)
                const int hd = a.ring_head[q];
                const int at = (hd >= 0 && hd < ring_n) ? hd : 0;
                a.ring[(size_t)q * (size_t)a.ring_cap + at] = (long long)token;
                a.ring_head[q] = (at + 1) % ring_n;
                const int f = a.ring_filled[q];
                a.ring_filled[q] = f < ring_n ? f + 1 : ring_n;
            }
            a.drawn_rw[q] += 1ull;
            if (a.stopped) a.stopped[r] = (a.stop_token && a.stop_token[q] == (long long)token) ? 1 : 0;
        }
        if (a.diag) { a.diag[4 * r] = dZ; a.diag[4 * r + 1] = dsum; a.diag[4 * r + 2] = dtarget; a.diag[4 * r + 3] = dp; }
    };
    if (c.status) { finish(); return; }

    CSTAMP(0);
#ifdef MOLLA_SAMPLE_TESTING
    if (a.prof && leader && c.tid == 0) {
        unsigned long long gt;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(gt));
        a.prof[(long long)r * 32 + 10] = (long long)gt; a.prof[(long long)r * 32 + 12] = blockIdx.x;
    }
#endif
    cluster_begun();
    // ---- 1. this block's range of the row, HBM -> shared memory
    const float *src = a.logits + lrow * a.row_stride + g.c0;
    const bool aligned = ((reinterpret_cast<uintptr_t>(src) & 15u) == 0);
    const int nbulk = aligned ? (g.nloc & ~3) : 0;
    if (c.tid == 0) {
        mbar_init(&A->mbar, 1);
        fence_proxy_async();
        if (nbulk > 0) {
            mbar_expect_tx(&A->mbar, (uint32_t)nbulk * 4u);
            for (int o = 0; o < nbulk; o += CL_PIECE)
                bulk_g2s_last_use(rowbuf + o, src + o, (uint32_t)min(CL_PIECE, nbulk - o) * 4u, &A->mbar);
        }
    }
    // meanwhile: this range's words of the grammar mask, where the tables will be
    unsigned int *mwords = reinterpret_cast<unsigned int *>(&A->u);
    static_assert(sizeof(A->u) >= (CL_CAPF / 32 + 2) * sizeof(unsigned int), "the mask's words fit");
    if (a.mask && g.nloc > 0) {
        const unsigned int *mrow = a.mask + (long long)r * a.mask_stride + (g.c0 >> 5);
        for (int i = c.tid; i < (((g.c0 & 31) + g.nloc + 31) >> 5); i += NT) mwords[i] = __ldg(mrow + i);
    }
    // and the tokens a bias or a penalty touches (sample.mojo:381-417), those of this range.
    // A small hash (keys and window counts) in the space the candidates use later.
    int *hkey = reinterpret_cast<int *>(A->cand);
    int *hcnt = hkey + HSLOTS;
    if (npatch > 0) {
        for (int i = c.tid; i < HSLOTS; i += NT) { hkey[i] = -1; hcnt[i] = 0; }
        __syncthreads();
        for (int i = c.tid; i < npatch; i += NT) {
            const bool is_bias = i < nb;
            const long long t64 = (is_bias ? a.bias_ids[b0 + i] : histp[i - nb]) - (long long)g.c0;
            if (t64 < 0 || t64 >= g.nloc) continue;
            const int tok = (int)t64;
            int s = hslot(tok);
            for (int probe = 0; probe < HSLOTS; probe++) {
                const int old = atomicCAS(&hkey[s], -1, tok);
                if (old == -1 || old == tok) { if (!is_bias) atomicAdd(&hcnt[s], 1); break; }
                s = (s + 1) & (HSLOTS - 1);
            }
        }
    }
    // what the bulk copies do not bring: the ragged end, or all of a row that is not 16-byte aligned
    for (int i = nbulk + c.tid; i < g.nloc; i += NT) rowbuf[i] = __ldg(src + i);
    for (int i = g.nloc + c.tid; i < NT * g.L; i += NT) rowbuf[i] = -INFINITY;
    __syncthreads();  // the barrier is initialised before anyone waits on it
    if (nbulk > 0) {
        bool done = false;
        for (int spin = 0; spin < (1 << 22); spin++) {
            if (mbar_try_wait(&A->mbar, 0u)) { done = true; break; }
        }
        if (!done) c.status |= MOLLA_ROW_LOAD_TIMEOUT;
    }
    if (MOLLA_KNOB(a, 16) && c.warp == 3) c.status |= MOLLA_ROW_LOAD_TIMEOUT;  // testing build: one warp reports a wait that ran out
    if (__syncthreads_or((c.status & MOLLA_ROW_LOAD_TIMEOUT) ? 1 : 0)) c.status |= MOLLA_ROW_LOAD_TIMEOUT;
    cluster_all_begun();
    CSTAMP(1);
    if (a.softcap > 0.0f) {
        const float rcap = softcap_plain(a.softcap) ? __frcp_rn(a.softcap) : 0.0f;
        for (int i = c.tid; i < g.nloc; i += 4 * NT) {
            float x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = i + u * NT < g.nloc ? rowbuf[i + u * NT] : 0.0f;
            softcap4(x, a.softcap, rcap);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (i + u * NT < g.nloc) rowbuf[i + u * NT] = x[u];
        }
        __syncthreads();
    }
    if (a.mask && g.nloc > 0) {
        // `_mask` (sample.mojo:371-379): what the grammar forbids is no candidate at all. A logit of
        // -inf is exactly that here: it wins no maximum, takes no bias or penalty that could bring it
        // back, its exponential is zero, and zeros are absent from every sum, count and walk.
        const int shift = g.c0 & 31;   // (a multiple of four: four logits' bits are in one word)
        for (int i = 4 * c.tid; i < g.nloc; i += 4 * NT) {
            const unsigned int w = mwords[(shift + i) >> 5] >> ((shift + i) & 31);
            float4 &x = *reinterpret_cast<float4 *>(rowbuf + i);
            x = make_float4((w & 1u) ? x.x : -INFINITY, (w & 2u) ? x.y : -INFINITY, (w & 4u) ? x.z : -INFINITY, (w & 8u) ? x.w : -INFINITY);
        }
        __syncthreads();
    }
    if (npatch > 0) {
        for (int s = c.tid; s < HSLOTS; s += NT) {
            const int tok = hkey[s];
            if (tok < 0) continue;
            float v = rowbuf[tok];
            for (int bq = 0; bq < nb; bq++)  // duplicates add up, in the order they were given
                if (a.bias_ids[b0 + bq] == (long long)tok + g.c0) v = __fadd_rn(v, a.bias_vals[b0 + bq]);
            const int n = hcnt[s];
            if (n > 0) {
                if (v > 0.0f) v = __fdiv_rn(v, rp);
                else v = __fmul_rn(v, rp);
                v = __fsub_rn(v, __fmul_rn((float)n, fp));
                v = __fsub_rn(v, pp);
            }
            rowbuf[tok] = v;
        }
        __syncthreads();
    }

    CSTAMP(2);
    // ---- 2. the maximum and its first index (kernel.mojo:571-585, sample.mojo:342-346)
    const long long n_lim = (k > 0 && k < a.V) ? (long long)k : (long long)a.V;
    const bool sampled = !greedy && n_lim > 1;  // rows that need more than the maximum
    const bool topp_on = (P < 1.0f) && (n_lim > 1);
    const bool pure = !topp_on && n_lim == (long long)a.V;
    const int i0 = c.tid * g.L;
    float tmax;
    int tj;
    {
        // four interleaved runs over the thread's range, each keeping its first maximum
        float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
        int j0 = 0, j1 = 1, j2 = 2, j3 = 3;
        int j = 0;
        for (; j + 4 <= g.L; j += 4) {
            const float x0 = rowbuf[i0 + j], x1 = rowbuf[i0 + j + 1], x2 = rowbuf[i0 + j + 2], x3 = rowbuf[i0 + j + 3];
            if (x0 > m0) { m0 = x0; j0 = j; }
            if (x1 > m1) { m1 = x1; j1 = j + 1; }
            if (x2 > m2) { m2 = x2; j2 = j + 2; }
            if (x3 > m3) { m3 = x3; j3 = j + 3; }
        }
        for (; j < g.L; j++) {
            const float x0 = rowbuf[i0 + j];
            if (x0 > m0) { m0 = x0; j0 = j; }
        }
        tmax = m0; tj = j0;
        if (m1 > tmax || (m1 == tmax && j1 < tj)) { tmax = m1; tj = j1; }
        if (m2 > tmax || (m2 == tmax && j2 < tj)) { tmax = m2; tj = j2; }
        if (m3 > tmax || (m3 == tmax && j3 < tj)) { tmax = m3; tj = j3; }
    }
    float cmax = tmax;
    int cidx = g.c0 + i0 + tj;
    block_argmax(c, cmax, cidx);
    int ceq = 0;
    if (!greedy && n_lim == 1) {
        // only a top-k of one asks how many share the maximum (the sort's first element is one of them)
        int e = 0;
        for (int j = 0; j < g.L; j++) e += (i0 + j < g.nloc && rowbuf[i0 + j] == cmax) ? 1 : 0;
        (void)block_excl_scan<int>(e, A->wsi, &ceq);
    }
    // A lower bound of the running sum before every thread's range: each range adds at least the
    // exponential of its own maximum. Relative to this block's maximum for now; the others' are
    // not known yet.
    float et = 0.0f, eex = 0.0f, etot = 0.0f;
    if (sampled) {
        if (i0 < g.nloc && tmax > -INFINITY) {
            const float d = __fsub_rn(tmax, cmax);
            et = expf_pinned((T == 1.0f) ? d : __fdiv_rn(d, T));
        }
        eex = block_excl_scan<float>(et, A->wsf, &etot);
        if (!pure) {
            // the head's threshold comes from the threads' maxima: how many lie how far below the maximum
            A->thist[c.tid] = 0u;
            __syncthreads();
            if (i0 < g.nloc) {
                const float dd = __fmul_rn(__fsub_rn(cmax, tmax), TRES);
                const int b = (dd >= 0.0f && dd < (float)(TBINS - 1)) ? (int)dd : TBINS - 1;
                sred_add(&A->thist[b], 1u);
            }
        }
    }
    __syncthreads();
    if (c.tid < g.G) {
        AuxC *ox = cl.map_shared_rank(A, c.tid);
        ox->x1_max[g.rank] = cmax; ox->x1_idx[g.rank] = cidx; ox->x1_eq[g.rank] = ceq; ox->x1_status[g.rank] = c.status;
        ox->x2_total[g.rank] = etot;
    }
    if (c.tid == 0) { A->ncand = 0; A->evt_thread = 0x7fffffff; }
    CSTAMP(13);
    cl.sync();
    float xmax = -INFINITY;
    int imax = 0x7fffffff, eqs = 0;
    for (int o = 0; o < g.G; o++) {
        c.status |= A->x1_status[o];
        const float m = A->x1_max[o];
        if (m > xmax) { xmax = m; imax = A->x1_idx[o]; eqs = A->x1_eq[o]; }
        else if (m == xmax) { imax = min(imax, A->x1_idx[o]); eqs += A->x1_eq[o]; }
    }
    if (imax == 0x7fffffff) imax = 0;
    if (c.status & MOLLA_ROW_LOAD_TIMEOUT) { finish(); return; }
    if (a.mask && !(xmax > -INFINITY)) { c.status |= MOLLA_ROW_EMPTY; finish(); return; }  // every candidate was filtered out

    CSTAMP(3);
    if (greedy) { token = imax; finish(); return; }
    if (n_lim == 1) {
        // top-k of one: the sort's first element is a maximum (sample.mojo:485-490)
        if (eqs > 1) c.status |= MOLLA_ROW_TOPK_TIE;
        token = imax; finish(); return;
    }

    const float top = (T == 1.0f) ? xmax : __fdiv_rn(xmax, T);
    const float u01 = draw01(a.seed ? a.seed[q] : 0ull, a.drawn ? a.drawn[q] : 0ull);
    const bool filter_ok = fabsf(top) < 1.0e5f;
    // how many the sorted head has to cover: top-k + 1 where a top-k is set (up to CL_HEAD_NEED: such
    // rows finish in the head), a fixed number where the nucleus alone ends the row
    const bool open_row = n_lim == (long long)a.V;
    long long need = open_row ? (long long)HEAD_NEED : n_lim + 1;
    if (need > CL_HEAD_NEED) need = CL_HEAD_NEED;
    if (need > a.V) need = a.V;

    // ---- 3. the bound relative to the row's maximum, and the head's threshold: a value that at
    // least `need` of the threads' maxima reach bounds the need-th largest element from below.
    float lb;
    {
        float lbbase = 0.0f, mine = 0.0f;
        for (int o = 0; o <= g.rank; o++) {
            const float d = __fsub_rn(A->x1_max[o], xmax);
            const float f = (A->x1_max[o] > -INFINITY) ? expf_pinned((T == 1.0f) ? d : __fdiv_rn(d, T)) : 0.0f;
            if (o < g.rank) lbbase += A->x2_total[o] * f; else mine = f;
        }
        lb = lbbase + eex * mine;
    }
    float tau_x = INFINITY;
    unsigned int tau_bits = 1u;
    if (!pure) {
        // thread t adds up, over the blocks, the counts of bin t of distance below the row's maximum
        // (a block's own bins are shifted by its maximum's distance, rounded up)
        int cnt = 0;
        for (int o = 0; o < g.G; o++) {
            const float dd = __fmul_rn(__fsub_rn(xmax, A->x1_max[o]), TRES);
            if (!(dd >= 0.0f && dd < (float)TBINS)) continue;
            const int lb_ = c.tid - (int)ceilf(dd);
            if (lb_ >= 0 && lb_ < TBINS - 1) cnt += (int)cl.map_shared_rank(A, o)->thist[lb_];
        }
        int tot;
        const int ex = block_excl_scan<int>(cnt, A->wsi, &tot);
        if ((long long)ex < need && (long long)(ex + cnt) >= need) A->evt_thread = c.tid;
        __syncthreads();
        const int gb = A->evt_thread;
        tau_x = (gb < TBINS - 1 && fabsf(xmax) < 65536.0f) ? __fsub_rn(xmax, __fmul_rn((float)(gb + 2), 1.0f / TRES)) : -INFINITY;
        const float tv = (T == 1.0f) ? tau_x : __fdiv_rn(tau_x, T);
        const unsigned int tb_ = __float_as_uint(expf_pinned(__fsub_rn(tv, top)));
        tau_bits = tb_ > 1u ? tb_ : 1u;
    }
    // what is below half an ulp of the bound is dropped; below top - 105 the exponential is
    // exactly zero whatever came before
    float mythr;
    {
        const float thr_rel = (filter_ok && lb > 0.0f) ? T * (top + logf(0.9f * lb) - REL_MARGIN) : -INFINITY;
        const float thr_zero = filter_ok ? T * (top - 105.0f) : -INFINITY;
        mythr = fminf(fmaxf(thr_rel, thr_zero), tau_x);
    }

    CSTAMP(4);
    // ---- 4. the second pass, in place: the exponential (temperature and softmax numerator,
    // sample.mojo:419-434) of what can matter, zero for the rest. Where a row's sum is still small
    // (its first columns) nearly everything matters, later almost nothing: the warps go through
    // the range in interleaved tiles, so that no warp is left alone with the dense stretch, and
    // evaluate what they keep in full warps.
    {
        static_assert(offsetof(AuxC, hidx) == offsetof(AuxC, pre) + sizeof(A->pre), "the head's candidates rely on this layout");
        static_assert(offsetof(AuxC, cand) == sizeof(A->u) && offsetof(AuxC, pc) == offsetof(AuxC, cand) + sizeof(A->cand) &&
                      sizeof(A->u) + sizeof(A->cand) >= (size_t)(NT + 4) * (CL_LMAX + 1),
                      "the threads' lists use the idle space of the tables and the candidates");
        static_assert(sizeof(A->pc) >= NWARP * CL_LMAX * sizeof(float) && sizeof(A->pre) >= NT * sizeof(float), "bounds per thread and per tile");
        unsigned long long *hcand = reinterpret_cast<unsigned long long *>(A->pre);  // CL_HEADC keys over pre + hidx
        auto value = [&](float xx) -> float {
            const float v = (T == 1.0f) ? xx : __fdiv_rn(xx, T);
            return expf_pinned_nonpos(__fsub_rn(v, top));  // no logit of the row exceeds its maximum
        };
        auto take = [&](unsigned int ebits, int i_block) {  // the head's candidates are picked up on the way
            if (!pure && ebits >= tau_bits) {
                const int pos = satom_add(&A->ncand, 1);
                if (pos < CL_HEADC) hcand[pos] = make_key(ebits, g.c0 + i_block);
            }
        };
        // Warp w takes the 32-wide tiles w, w + 16, w + 32, ... of the range, so the dense stretch
        // is spread evenly over all threads. A tile tests its elements against the lowest bound of
        // the threads it overlaps (keeping more than necessary is always right). Every thread notes
        // the tiles in which it keeps its element in a list of its own and evaluates the list
        // afterwards, four at a time: the lists of a warp's lanes are about equally long, and no
        // conversion, population count, bit search or atomic (all of which issue at a fraction of
        // the rate of the rest) is needed to build them.
        unsigned char *klist = reinterpret_cast<unsigned char *>(&A->u);  // [entry][thread], over u + cand
        float *thr_t = A->pc;  // a bound per tile
        {
            float *thr_s = A->pre;  // every thread's bound
            thr_s[c.tid] = mythr;
            __syncthreads();
            // (x / L without a division: exact for x < 2^32 / L, and x stays below NT * L)
            const unsigned int l_magic = (unsigned int)((0x100000000ull + (unsigned long long)g.L - 1ull) / (unsigned long long)g.L);
            for (int t = c.tid; t < NWARP * g.L; t += NT) {
                const int o0 = (int)__umulhi((unsigned int)(32 * t), l_magic), o1 = min(NT - 1, (int)__umulhi((unsigned int)(32 * t + 31), l_magic));
                float m = thr_s[o0];
                for (int o = o0 + 1; o <= o1; o++) m = fminf(m, thr_s[o]);
                thr_t[t] = m;
            }
            __syncthreads();
        }
        CSTAMP(16);
        constexpr int KSTRIDE = NT + 4;  // bytes per list entry row: rows start one bank apart
        int cnt = 0;
        {
            unsigned char *kp = klist + c.tid;  // where this thread's next entry goes
            auto take_tile = [&](int k, int p, float x, float th) {
                // no branch: the entry is written in any case and stays only if the element is kept
                const bool keep = x >= th;
                *kp = (unsigned char)k;
                kp += keep ? KSTRIDE : 0;
                cnt += keep ? 1 : 0;
                rowbuf[p] = keep ? x : 0.0f;
            };
            int k = 0;
            for (; k + 4 <= g.L; k += 4) {  // four tiles' loads ahead of their stores
                int p[4];
                float x[4], th[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int t = (k + u) * NWARP + c.warp;
                    p[u] = (t << 5) + c.lane;
                    x[u] = rowbuf[p[u]];
                    th[u] = thr_t[t];
                }
#pragma unroll
                for (int u = 0; u < 4; u++) take_tile(k + u, p[u], x[u], th[u]);
            }
            for (; k < g.L; k++) {
                const int t = k * NWARP + c.warp;
                const int p = (t << 5) + c.lane;
                take_tile(k, p, rowbuf[p], thr_t[t]);
            }
        }
        CSTAMP(18);
        const int base = (c.warp << 5) + c.lane;
        auto entry = [&](int i) { return (((int)klist[i * KSTRIDE + c.tid] * NWARP) << 5) + base; };
        int i = 0;
        for (; i + 4 <= cnt; i += 4) {  // (no predicates in here: they would turn into branches around every evaluation)
            int pos[4];
            float y[4];
#pragma unroll
            for (int u = 0; u < 4; u++) pos[u] = entry(i + u);
#pragma unroll
            for (int u = 0; u < 4; u++) y[u] = value(rowbuf[pos[u]]);
#pragma unroll
            for (int u = 0; u < 4; u++) { rowbuf[pos[u]] = y[u]; take(__float_as_uint(y[u]), pos[u]); }
        }
        for (; i < cnt; i++) {
            const int pos = entry(i);
            const float y = value(rowbuf[pos]);
            rowbuf[pos] = y;
            take(__float_as_uint(y), pos);
        }
        __syncthreads();
        CSTAMP(17);
        // the head's candidates to where the head looks for them
        const int nh = min(A->ncand, CL_HEADC);
        unsigned long long mine[(CL_HEADC + NT - 1) / NT];
#pragma unroll
        for (int u = 0; u < (CL_HEADC + NT - 1) / NT; u++) mine[u] = (c.tid + u * NT < nh) ? hcand[c.tid + u * NT] : 0ull;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < (CL_HEADC + NT - 1) / NT; u++)
            if (c.tid + u * NT < nh) A->cand[c.tid + u * NT] = mine[u];
    }
    __syncthreads();
    CSTAMP(5);
    // how many candidates for the head every block holds
    if (c.tid < g.G) cl.map_shared_rank(A, c.tid)->x3_n[g.rank] = A->ncand;

    // ---- 5. the softmax denominator, exactly as the sequential loop rounds it
    const ClSum zs = cluster_exact_sum(A, g, a.Vc, a.V, rowbits, CPROF_SLOTS(leader, 14));
    const float Z = zs.s;
    if (zs.slow) c.status |= MOLLA_ROW_SLOW_PATH;
    dZ = Z;

    CSTAMP(6);

    // min-p (sample.mojo:508-523): see the note at the same place in sample_rows_kernel
    long long n_use = n_lim;
    const bool typ_on = typ < 1.0f;
    unsigned int minp_pbits = 0u;
    if (minp > 0.0f) {
        const float p_top = __fdiv_rn(expf_pinned(__fsub_rn(top, top)), Z);
        const float floor_p = __fmul_rn(p_top, minp);
        minp_pbits = __float_as_uint(floor_p);
        if (!(floor_p >= 2.2e-8f)) {
            c.status |= MOLLA_ROW_UNSUPPORTED;
        } else if (!pure) {
            unsigned int lo_b = 0u, hi_b = 0x3F800000u;
            for (int it = 0; it < 32 && lo_b < hi_b; it++) {
                const unsigned int mid = lo_b + ((hi_b - lo_b) >> 1);
                if (__fdiv_rn(__uint_as_float(mid), Z) >= floor_p) hi_b = mid; else lo_b = mid + 1u;
            }
            const unsigned int e_floor = hi_b;
            int cnt_ge = 0;
            for (int i = c.tid; i < g.nloc; i += NT) cnt_ge += (rowbits[i] >= e_floor && rowbits[i] != 0u) ? 1 : 0;
            int n_ge_loc;
            (void)block_excl_scan<int>(cnt_ge, A->wsi, &n_ge_loc);
            if (c.tid < g.G) cl.map_shared_rank(A, c.tid)->x4_n[g.rank] = n_ge_loc;
            cl.sync();
            long long n_ge = 0;
            for (int o = 0; o < g.G; o++) n_ge += A->x4_n[o];
            if (n_ge < 1) n_ge = 1;  // never empties
            if (n_ge < n_use) n_use = n_ge;
        }
    }
    if (c.status & MOLLA_ROW_UNSUPPORTED) { finish(); return; }

    if (pure) {
        // ---- 6a. nothing sorted: the draw walks the vocabulary in order (sample.mojo:365-369,
        // 580-594): probabilities p = e / Z (:437-438), what min-p drops becomes zero
        for (int i = c.tid; i < g.nloc; i += NT) {
            const unsigned int eb = rowbits[i];
            if (eb == 0u) continue;
            unsigned int pb = __float_as_uint(__fdiv_rn(__uint_as_float(eb), Z));
            if (pb < minp_pbits) pb = 0u;
            rowbits[i] = pb;
        }
        const ClSum s1 = cluster_exact_sum(A, g, a.Vc, a.V, rowbits);
        const float sum = s1.s;
        const float target = __fmul_rn(u01, sum);
        const int drawn = cluster_locate(A, g, a.Vc, a.V, rowbits, sum, target);
        if (s1.slow) c.status |= MOLLA_ROW_SLOW_PATH;
        dsum = sum; dtarget = target;
        if (drawn >= 0) token = drawn;
        else {
            // the walk fell off the end: the reference returns the last token of the vocabulary,
            // whether or not it could matter to any sum ... or the last one min-p left
            token = a.V - 1;
            if (minp_pbits) {
                int last = -1;
                for (int i = c.tid; i < g.nloc; i += NT)
                    if (rowbits[i] >= minp_pbits && rowbits[i] != 0u) last = max(last, g.c0 + i);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
                __syncthreads();
                if (c.lane == 0) A->wsi[c.warp] = last;
                __syncthreads();
                if (c.tid < g.G) {
                    int m = -1;
                    for (int w = 0; w < NWARP; w++) m = max(m, A->wsi[w]);
                    cl.map_shared_rank(A, c.tid)->x4_n[g.rank] = m;
                }
                cl.sync();
                last = -1;
                for (int o = 0; o < g.G; o++) last = max(last, A->x4_n[o]);
                token = last >= 0 ? last : imax;
            }
        }
        finish();
        return;
    }

    CSTAMP(7);
    // ---- 6b. sorted order. The head's candidates go to the leader as probabilities.
    int nc_tot = 0, cbase = 0;
    bool head_overflow = false;
    for (int o = 0; o < g.G; o++) {
        const int n = A->x3_n[o];
        if (o < g.rank) cbase += n;
        nc_tot += n;
        if (n > CL_HEADC) head_overflow = true;
    }
    if (nc_tot > CL_HEADC) head_overflow = true;
    if (!head_overflow) {
        const int mine = A->x3_n[g.rank];
        for (int i = c.tid; i < mine; i += NT) {
            const unsigned long long kk = A->cand[i];
            const unsigned long long nk = ((unsigned long long)__float_as_uint(__fdiv_rn(key_val(kk), Z)) << 32) | (kk & 0xFFFFFFFFull);
            if (leader) A->cand[i] = nk; else lead->cand[cbase + i] = nk;
        }
    }
    cl.sync();
    int nc = head_overflow ? 0 : nc_tot;
    unsigned int tau_head = 0xFFFFFFFFu;
    if (head_overflow) c.status |= MOLLA_ROW_SLOW_PATH;  // no head: the descending walk takes everything from the top
    if (leader) {
        // (sorted through the tables' space and, where there are many, that of pc and pre)
        static_assert(CL_HEADC <= NC && sizeof(A->u) >= NBINS * sizeof(unsigned int) &&
                      offsetof(AuxC, pre) == offsetof(AuxC, pc) + sizeof(A->pc) && sizeof(A->pc) + sizeof(A->pre) >= CL_HEADC * sizeof(unsigned long long), "room for the sort");
        sort_keys<NT, 256>(nc, A->cand, reinterpret_cast<unsigned long long *>(A->pc), A->pc, A->u.h.hq, reinterpret_cast<unsigned int *>(A->wsi), reinterpret_cast<unsigned int *>(A->wsf));
#ifdef MOLLA_SAMPLE_TESTING
        if (a.topk_out) {
            for (int i = c.tid; i < a.topk_cap; i += NT)
                a.topk_out[(long long)r * a.topk_cap + i] = (i < nc && (long long)i < n_use) ? key_idx(A->cand[i]) : -1;
        }
#endif
        if (c.warp == 0) {
            const HeadEnd e = head_end(HeadRule{n_lim, P, open_row, topp_on, typ_on}, a.V, A->pc, A->pre, nc, nc, n_use, false, head_overflow, u01);
            if (c.lane == 0) {
                A->b_s = e.s; A->b_pos = e.pos; A->b_event = EV_NONE; A->b_idx = -1; A->b_p = 0.0f; A->b_aux = (int)e.tie;
                if (typ_on) A->ncand = e.cut;  // the typical-p filter takes over from here
                if (e.at >= 0) { A->b_event = EV_DRAW; A->b_idx = key_idx(A->cand[e.at]); A->b_p = A->pc[e.at]; A->b_sum = e.sum; A->b_target = e.target; }
            }
        } else {   // what the walks behind the head ask of it
            for (int i = c.tid - 32; i < nc; i += NT - 32) {
                const float p = A->pc[i];
                const bool eq = (i > 0 && A->pc[i - 1] == p) || (i + 1 < nc && A->pc[i + 1] == p);
                A->hidx[i] = (unsigned int)key_idx(A->cand[i]) | (eq ? 0x80000000u : 0u);
            }
        }
        __syncthreads();
        c.status |= (unsigned int)A->b_aux;
        const float head_s = A->b_s;
        const long long head_pos = A->b_pos;
        int kind = 1;  // 0: the row is finished; 1: past the head
        if (typ_on) {
            const int m = A->ncand;
            if (m <= 0 || m > HEADC) {
                c.status |= MOLLA_ROW_UNSUPPORTED;  // what the earlier filters left reaches past the head, or is wider than the filter's scratch
            } else {
                typical_head(c, m, typ, u01);
                token = A->b_idx; dp = A->b_p; dsum = A->b_sum; dtarget = A->b_target;
                c.status |= (unsigned int)A->b_aux;
            }
            kind = 0;
        } else if (A->b_event == EV_DRAW) {
            token = A->b_idx; dp = A->b_p; dsum = A->b_sum; dtarget = A->b_target;
            kind = 0;
        }
        __syncthreads();
        if (c.tid < g.G) {
            AuxC *ox = cl.map_shared_rank(A, c.tid);
            ox->r_kind = kind; ox->r_s = head_s; ox->r_pos = head_pos; ox->r_status = c.status;
        }
    }
    cl.sync();
    if (A->r_kind == 0) { finish(); return; }
    c.status |= A->r_status;
    const float head_s = A->r_s;
    const long long head_pos = A->r_pos;

    CSTAMP(8);
    // ---- 7. past the head: the cut walk, then the draw walk, over the probabilities
    // (sample.mojo:437-438); what the head took is consumed
    for (int i = c.tid; i < g.nloc; i += NT) {
        const unsigned int eb = rowbits[i];
        if (eb == 0u) continue;
        unsigned int pb = __float_as_uint(__fdiv_rn(__uint_as_float(eb), Z));
        if (!head_overflow && eb >= tau_bits) pb = 0u;
        rowbits[i] = pb;
    }
    __syncthreads();
    // One call site for both walks (the walk is most of this kernel's code, and what a row runs
    // through has to stay in the instruction cache): leg 0 is the cut walk, leg 1 the draw walk.
    const bool limited = n_use < (long long)a.V;
    ClWalk w;
    ClResume resume;
    resume.valid = 0;
    int cut_event = EV_NONE, cut_idx = -1;
    float cut_p = 0.0f, sum = 0.0f, target = 0.0f;
    bool settled = false;    // the token is known, or the row is degenerate
    bool resolved = false;
    for (int leg = 0; leg < 2; leg++) {
        w.s = head_s; w.pos = head_pos; w.tau = tau_head;
        w.event = EV_NONE; w.idx = -1; w.p = 0; w.tie = 0;
        const bool cut_round = leg == 0;
        descend_cluster(cl, c, g, rowbits, w, (cut_round && topp_on) ? P : 3.4e38f, cut_round ? 3.4e38f : target,
                        (cut_round && limited) ? n_use : -1, resume, !cut_round, cut_round ? CPROF_SLOTS(leader, 20) : nullptr);
        if (!cut_round) {
            if (w.event == EV_DRAW) {
                token = w.idx; dp = w.p; resolved = true;
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
        cl.sync();
        if (leader) {  // is the drawn element in the head? (the first prefix sum above the target)
            if (c.tid == 0) A->evt_thread = 0x7fffffff;
            __syncthreads();
            for (int i = c.tid; i < nc; i += NT)
                if (target < A->pre[i]) { atomicMin(&A->evt_thread, i); break; }
            __syncthreads();
        }
        if (leader && c.tid == 0) {
            const int at = (A->evt_thread == 0x7fffffff) ? -1 : A->evt_thread;
            int ev = EV_NONE, idx = -1, aux = 0;
            float pv = 0.0f;
            if (at >= 0) {
                ev = EV_DRAW; idx = (int)(A->hidx[at] & 0x7fffffffu);
                pv = __fsub_rn(A->pre[at], at > 0 ? A->pre[at - 1] : 0.0f);
                aux = (A->hidx[at] & 0x80000000u) ? MOLLA_ROW_CHOSEN_TIE : 0;
            }
            for (int o = 0; o < g.G; o++) {
                AuxC *ox = cl.map_shared_rank(A, o);
                ox->r_kind = ev; ox->r_idx = idx; ox->r_s = pv; ox->r_status = (unsigned int)aux;
            }
        }
        cl.sync();
        if (A->r_kind == EV_DRAW) {
            token = A->r_idx; dp = A->r_s; c.status |= A->r_status;
            settled = true;
            break;
        }
        if (!(target < sum)) break;
    }
    if (!settled) {
        {
            if (!resolved) {
                // the walk falls off the end: the last kept candidate (sample.mojo:591-594)
                if (cut_event == EV_CUT || cut_event == EV_LIMIT) {
                    token = cut_idx; dp = cut_p;
                } else {
                    // everything listed was kept: its smallest value, highest id last
                    unsigned long long best = ~0ull;
                    for (int i = c.tid; i < g.nloc; i += NT) {
                        const unsigned int pb = rowbits[i];
                        if (pb == 0u) continue;
                        const unsigned long long kk = make_key(pb, g.c0 + i);
                        best = kk < best ? kk : best;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                        best = ob < best ? ob : best;
                    }
                    __syncthreads();
                    if (c.lane == 0) A->wsu[c.warp] = best;
                    __syncthreads();
                    if (c.tid < g.G) {
                        unsigned long long m = A->wsu[0];
                        for (int v = 1; v < NWARP; v++) m = A->wsu[v] < m ? A->wsu[v] : m;
                        cl.map_shared_rank(A, c.tid)->x5_key[g.rank] = m;
                    }
                    cl.sync();
                    best = ~0ull;
                    for (int o = 0; o < g.G; o++) best = A->x5_key[o] < best ? A->x5_key[o] : best;
                    token = (best != ~0ull) ? key_idx(best) : imax;
                }
            }
        }
    }
    finish();
}

// How a vocabulary of V logits is laid over a cluster: blocks per cluster (0 = too wide), logits
// per block (a multiple of four: bulk copies start on 16-byte boundaries) and logits per thread
// (odd: conflict-free shared-memory strides).
struct ClusterShape { int G, Vc, L; };

// The smallest cluster that holds the row; for a batch so small that larger clusters of all
// its rows are still resident together (a lone decode stream, a few rows per GPU), the largest
// such cluster: the passes over the row shorten with the range, and nobody waits for an SM.
ClusterShape cluster_shape(int V, int B, int sms) {
    ClusterShape best{0, 0, 0};
    for (int G = 1; G <= CL_MAX_G; G *= 2) {
        const int Vc = ((((V + G - 1) / G) + 3) / 4) * 4;
        int L = (Vc + NT - 1) / NT;
        if ((L & 1) == 0) L += 1;
        if (L > CL_LMAX) continue;
        if (best.G == 0) { best = ClusterShape{G, Vc, L}; continue; }
        // (clusters do not fill every SM: leave the same margin the resident-cluster count shows)
        if ((long long)B * G * 9 <= (long long)sms * 8 && L >= 9) best = ClusterShape{G, Vc, L};
    }
    return best;
}

constexpr size_t CL_SMEM = (size_t)CL_CAPF * 4 + ((sizeof(AuxC) + 15) / 16) * 16;
constexpr int CL_MAX_DEVICES = 64;

void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, unsigned int blocks, int G, cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(blocks); cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = CL_SMEM; cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)G; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
}

// How many clusters of G of the kernel's blocks this device holds at a time (asked once per device and size).
int clusters_resident(int dev, int G) {
    static int known[CL_MAX_DEVICES][CL_MAX_G + 1] = {};  // 0 unknown, -1 none
    if (dev < 0 || dev >= CL_MAX_DEVICES) return 0;
    if (known[dev][G]) return known[dev][G] > 0 ? known[dev][G] : 0;
    int n = 0;
    bool ok = cudaFuncSetAttribute(sample_rows_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM) == cudaSuccess;
    if (ok) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        cluster_config(cfg, at, (unsigned)G, G, nullptr);
        ok = cudaOccupancyMaxActiveClusters(&n, sample_rows_cluster_kernel, &cfg) == cudaSuccess && n > 0;
    }
    if (!ok) (void)cudaGetLastError();
    known[dev][G] = ok ? n : -1;
    return ok ? n : 0;
}

}  // namespace

bool molla_cluster_is_block(int V) { return V <= CL_CAPF; }

// A row in the shared memory of its cluster is worked on in one launch, so as long as the clusters of all rows are
// resident together the call is one row long: 32 rows of 8000 to 151936 logits take 6 to 8 us if greedy, 28 to 43
// with a top-k of 40, 33 to 74 with mixed settings, 48 to 92 with a nucleus, 36 to 69 where nothing is sorted (the
// tile kernels: 11 to 14, 36 to 51, 51 to 78, 45 to 110, 57 to 82; all in CUDA graphs). A second round of clusters doubles that and the
// tile kernels pass it: 128 rows of 73000 with a top-k 59 against 76 us, nothing sorted 102 against 125; 256 rows of
// 8000 with a top-k 44 against 52, a nucleus 58 against 90. Two kinds of batch the line cuts wrong, and as the
// settings are on the device it cannot see them: up to 512 rows of 2500 to 20000 logits, each with its own settings
// (256 of 8000: 95 us in tiles, 64 in clusters), and rows that all ask for a wide top-k (64 of 50257: 192 in clusters,
// 63 in tiles).
bool molla_cluster_better(int V, int B, int call_B) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const ClusterShape cs = cluster_shape(V, call_B, sms);
    return cs.G != 0 && (long long)B * cs.G * 9 <= (long long)sms * 8 && clusters_resident(dev, cs.G) > 0;
}

// Whether the clusters of all B rows fit the device at the same time, where it matters. Of those of eight blocks 15 or 16
// fit, depending on which of its SMs a device has. Where it is 15, 16 rows take two rounds of clusters: whatever the length, calls
// whose rows are all alike are then better off in the tile kernels, while mixed settings, of which the row that starts
// late is seldom the dearest, are not (clusters / tiles, us): 151936 logits, a top-k of 40 67 / 48, a nucleus 134 / 120, nothing
// sorted 97 / 79, mixed 82 / 99; 235000 72 / 53, 156 / 129, 115 / 84, 96 / 108; 262144 76 / 53, 160 / 129, 122 / 83, 103 / 107;
// 290000 77 / 58, 168 / 131, 122 / 85, 107 / 109. A row's time in a cluster grows with its length and the tile
// kernels' hardly does, so from 240000 on mixed rows lose next to nothing. With a softcap, of which the tile kernels do
// every logit twice, they do (262144: 117 / 124), and stay.
constexpr int TWO_ROUNDS_V = 240000;
bool molla_cluster_resident(int V, int B, int call_B, bool capped) {
    if (capped || V <= TWO_ROUNDS_V) return true;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const ClusterShape cs = cluster_shape(V, call_B, sms);
    return cs.G != 0 && B <= clusters_resident(dev, cs.G);
}

int molla_cluster_launch(const BatchArgs &args_in, cudaStream_t st, char *err, size_t errlen) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    BatchArgs a = args_in;
    const ClusterShape cs = cluster_shape(a.V, a.layout_B > 0 ? a.layout_B : a.B, sms);
    a.G = cs.G; a.Vc = cs.Vc; a.L = cs.L;
    a.Vg = a.V; a.col0 = 0; a.mode = 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, (unsigned)a.B * (unsigned)cs.G, cs.G, st);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, sample_rows_cluster_kernel, a);
    if (e != cudaSuccess) {
        snprintf(err, errlen, "kernel launch failed: %s", cudaGetErrorString(e));
        return MOLLA_ERR_CUDA;
    }
    return MOLLA_OK;
}
