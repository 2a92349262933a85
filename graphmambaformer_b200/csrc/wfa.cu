// Unit-cost global wavefront alignment (edit distance + CIGAR).
//
// Semantics (graphmambaformer/alignment/extension.py L308-463,
// WavefrontAligner): diagonal k = i - j, offset = query bases consumed.
// Wavefront 0 is the match run from (0, 0); wavefront s takes, per diagonal
// k in [-s, s], the largest of three candidates of wavefront s-1 --
// substitution (k, +1), insertion (k-1, +1), deletion (k+1, +0) -- each
// rejected on its own when it leaves the matrix (offset outside [0, n] or
// column outside [0, m]), then extends through the run of matching codes (a
// code matches iff equal, >= 0 and != 5).  The alignment is complete at the
// first s whose diagonal n - m reaches n; the distance bound is tested after
// that check, so a pair exactly at the bound succeeds.  n == 0 or m == 0 is
// answered directly (distance max(n, m), CIGAR I n D m).  The traceback walks
// back from (s, n - m), taking at each score the first largest of the
// unclipped candidates X, I, D; the gap between that candidate and the
// diagonal's reach is a run of matches (never negative).
//
// Layout:
//   forward kernel  persistent blocks pull pairs in the caller's order.  A pair
//                   is computed by one warp, or by the whole block when it is
//                   long (a side of 4000 codes, or distance 96 when it is
//                   known): the team's threads take the diagonals of a
//                   wavefront in turn and extend each one 4, then 8 codes per
//                   step, long runs 128 codes per step of their warp.
//                   The two live wavefronts sit in shared memory (scores up
//                   to 254 for a warp, 2,049 or 8,205 for a block) and move
//                   to a global slot beyond: one per block where its shared
//                   memory may not do, and 16-bit ones that the warps claim as
//                   they need them (a side of theirs is below 4000, so 148
//                   blocks of 32 warps need 152 MB for any bound, 64 pairs 2 MB;
//                   a 32-bit slot of the whole bound for every warp of every
//                   block took 311 and 134 MB at 4,096).  With a history, wavefront s is also
//                   stored, for the walk.
//   walk kernel     one warp per pair, from the last wavefront back.
//
// What bounds it is the critical path: a 20 kb ONT-like pair takes ~1,000
// wavefronts one after another, whatever else the GPU does.  So a long pair's
// block has 1,024 threads (a wavefront of 2s+1 diagonals in few turns), a turn
// compares 4 or 8 codes at once with 32-bit word indices, and the history is
// kept while the distance is found (in chunks of 32 wavefronts, allocated as
// the pair goes) instead of replaying every pair to its known distance.  A run
// of more than 20 matches is finished by the diagonal's whole warp.  Measured
// on one B200, 4,000 mixed pairs of 150-20,000 bases: forward 3,711 + 4,061 us
// (distance, then replay with history) -> 1,654 us, with the warps' runs 1,340
// us; walk 1,091 -> 281 us.

#include <algorithm>

#include "gmf_common.cuh"

namespace {

constexpr int WFA_SMEM_S = 254;                       // a warp's wavefronts up to this score in shared memory
constexpr int WFA_SMEM_WF = 2 * WFA_SMEM_S + 5;       // ints per shared wavefront (two sentinels at each end)
constexpr int WFA_NONE = -(1 << 30);                  // no offset: stays negative after the + 1 of a candidate
constexpr int WFA_NONE16 = -(1 << 14);                // the same in 16 bits
constexpr int WFA_LONG_LEN = 4000;  // distance unknown: a pair with a side this long gets a whole block
constexpr int WFA_LONG_D = 96;      // distance known: a pair at this distance gets a whole block
constexpr int WFA_WIDE = 1024;      // threads of a block when its wavefronts always fit its shared memory
constexpr int WFA_NARROW = 256;     // and beyond
constexpr int WFA_CHUNK = 32;       // wavefronts per history chunk

__host__ __device__ constexpr int block_scores(int threads) { return (threads / 32 * WFA_SMEM_WF - 5) / 2; }

struct Seq {
    const uint32_t* w;  // aligned words covering the whole buffer
    int nw;
    long long base;     // byte offset of the buffer's first code from w
};

__host__ __device__ inline Seq make_seq(const int8_t* buf, long long total) {
    Seq s;
    const uintptr_t a = (uintptr_t)buf & ~(uintptr_t)3;
    s.w = reinterpret_cast<const uint32_t*>(a);
    s.base = (long long)((uintptr_t)buf - a);
    const long long nw = total > 0 ? ((s.base + total - 1) >> 2) + 1 : 1;
    s.nw = nw > 0x7fffffffll ? 0x7fffffff : (int)nw;
    return s;
}

// One sequence of a pair: words from the one that holds its first code on.
// Words beyond the buffer are clamped; they only feed codes past the end.
struct Codes {
    const uint32_t* w;
    int last;   // last word that may be read
    int shift;  // codes before the first one in word 0
    __device__ Codes(const Seq& s, long long first) {
        const long long at = s.base + first;
        long long wi = at >> 2;
        if (wi >= s.nw) wi = s.nw - 1;  // an empty sequence at the buffer's end
        w = s.w + wi;
        last = s.nw - 1 - (int)wi;
        shift = (int)(at & 3);
    }
    __device__ unsigned ld(int i) const { return __ldg(w + min(i, last)); }
};

struct WfaArgs {
    int n_pairs;
    const long long* q_off;
    const long long* t_off;
    const int* order;
    Seq Q, T;
    int max_distance;
    int eff;               // largest distance any pair can reach: min(max_distance, longest side)
    int warp_eff;          // the same for a pair of one warp
    int* block_spill;      // 2 * (2*eff + 5) ints per block, or null where its shared memory holds every score
    short* warp_spill;     // slots of 2 * (2*warp_eff + 5), or null when warp_eff <= WFA_SMEM_S
    unsigned* warp_slots;  // slots claimed
    unsigned* work;        // pair counters of the forward and the walk kernel
    int* distance;         // written, or read when the history is replayed (KNOWN)
    int* hist;
    long long hist_cap;    // ints
    unsigned long long* hist_used;
    long long* hist_off;   // per pair: offset of its history (KNOWN) or of its last chunk, -1 when absent
    int* err;
    int long_len, long_d;  // whole-block pairs: a side of long_len codes, or (KNOWN) distance long_d
};

// How a forward pass keeps wavefronts.
enum Mode {
    DIST = 0,    // not at all: the distance alone
    KNOWN = 1,   // distance known: wavefront s at s*s + s + k of (d+1)^2 ints
    CHUNKED = 2  // distance unknown: chunks of 32 wavefronts, each behind the offset of the one before
};

// Chunk c holds wavefronts [32c, 32c + 32), wavefront s at s*s - (32c)^2 + s + k
// behind 2 ints of link.
__device__ __forceinline__ long long chunk_ints(int c) { return 2 + (long long)WFA_CHUNK * WFA_CHUNK * (2 * c + 1); }
__device__ __forceinline__ long long chunk_row(int s) {
    const long long s0 = s & ~(WFA_CHUNK - 1);
    return 2 + (long long)s * s - s0 * s0;
}

// Chunks of a pair's own share of the history: those of about 8% differences,
// as the caller sizes the workspace.
__device__ __forceinline__ int history_share(int longest, int bound) {
    return min(min(longest, bound), (int)(longest * 8ll / 100) + 48) / WFA_CHUNK + 1;
}

// The place of a pair's chunk c in the history, or -1 when it does not fit.
// A pair takes its own share as long as there is room, and more only while
// half of the room is left, so that a few unrelated pairs do not use up the
// others' shares (160 of 4.1 kb before 64 related ones of 300 bases, in a
// workspace of their shares: the 64 found nothing left).  A chunk that does
// not fit gives its place back, for smaller ones: the one request that crosses
// the end sets the counter back, every other one until then starts beyond the
// end and is refused.  (Taken by compare and swap instead, one chunk at a
// time, the 4,000 first chunks alone cost 3 ms.)
__device__ __forceinline__ long long take_chunk(const WfaArgs& A, int c, int own) {
    const long long need = chunk_ints(c);
    if (c >= own && (long long)*(volatile unsigned long long*)A.hist_used + need > A.hist_cap / 2) return -1;
    const long long o = (long long)atomicAdd(A.hist_used, (unsigned long long)need);
    if (o + need <= A.hist_cap) return o;
    if (o <= A.hist_cap) atomicExch(A.hist_used, (unsigned long long)o);
    return -1;
}

// Bytes of a that match nothing (N = 5, negative), as their top bits; those
// above the lowest may be false.
__device__ __forceinline__ unsigned unmatched(unsigned a) {
    const unsigned y = a ^ 0x05050505u;  // a zero byte is an N
    return (((y - 0x01010101u) & ~y) | a) & 0x80808080u;
}

// The two sequences of a pair.  plain: no code of the query is an N or
// negative, so equal codes match.
struct Pair {
    Codes Q, T;
    int n, m;
    bool plain;
    __device__ Pair(const Seq& sq, long long q0, int n_, const Seq& st, long long t0, int m_)
        : Q(sq, q0), T(st, t0), n(n_), m(m_), plain(false) {}
    // Lowest set bit in the first of 4 codes that differs or matches nothing; 0 when all match.
    __device__ unsigned differing(unsigned a, unsigned b) const {
        const unsigned x = a ^ b;
        return plain ? x : x | unmatched(a);
    }
};

// Offset after the run of matches from query position i on diagonal k, from
// aligned words of both sequences: 4 codes (most diagonals stop there), then
// 8 at a time up to WFA_SHORT codes; `more` when the run goes on (limits of 4,
// 12, 20 and 28 codes: 2,299 / 2,224 / 2,209 / 2,245 us for the 4,000 pairs).
constexpr int WFA_SHORT = 20;
__device__ __forceinline__ int wfa_extend(const Pair& P, int i, int k, bool& more) {
    const int j = i - k;  // (j >= 0 for every offset i >= 0 of a wavefront)
    const int lim = min(P.n - i, P.m - j);
    if (lim <= 0) return i;
    int wq = (P.Q.shift + i) >> 2, wt = (P.T.shift + j) >> 2;
    const int sq = ((P.Q.shift + i) & 3) * 8, st = ((P.T.shift + j) & 3) * 8;
    unsigned q0 = P.Q.ld(wq), q1 = P.Q.ld(wq + 1), t0 = P.T.ld(wt), t1 = P.T.ld(wt + 1);
    unsigned x = P.differing(__funnelshift_r(q0, q1, sq), __funnelshift_r(t0, t1, st));
    if (x) return i + min((__ffs((int)x) - 1) >> 3, lim);
    int adv = 4;
    while (adv < lim && adv < WFA_SHORT) {
        ++wq;
        ++wt;
        q0 = q1;
        t0 = t1;
        const unsigned q2 = P.Q.ld(wq + 2), t2 = P.T.ld(wt + 2);
        q1 = P.Q.ld(wq + 1);
        t1 = P.T.ld(wt + 1);
        x = P.differing(__funnelshift_r(q0, q1, sq), __funnelshift_r(t0, t1, st));
        const unsigned y = P.differing(__funnelshift_r(q1, q2, sq), __funnelshift_r(t1, t2, st));
        if (x | y) return i + min(adv + (x ? (__ffs((int)x) - 1) >> 3 : 4 + ((__ffs((int)y) - 1) >> 3)), lim);
        adv += 8;
        ++wq;
        ++wt;
        q1 = q2;
        t1 = t2;
    }
    more = adv < lim;
    return i + min(adv, lim);
}

// The same by the whole warp, 128 codes at a time (i and k are the same in
// every lane).  Long runs are the few diagonals around the path: one lane
// would hold up its wavefront for as many steps as the longest of them takes
// (148 HiFi-like pairs of 15-20 kb: 528 us a call one lane at a time, 245 us
// so; the 4,000 mixed pairs 2,571 -> 2,209 us).
__device__ __forceinline__ int wfa_extend_warp(const Pair& P, int i, int k) {
    const int j = i - k, lim = min(P.n - i, P.m - j), lane = threadIdx.x & 31;
    int wq = ((P.Q.shift + i) >> 2) + lane, wt = ((P.T.shift + j) >> 2) + lane;
    const int sq = ((P.Q.shift + i) & 3) * 8, st = ((P.T.shift + j) & 3) * 8;
    for (int at = 0; at < lim; at += 128, wq += 32, wt += 32) {
        const unsigned q = __funnelshift_r(P.Q.ld(wq), P.Q.ld(wq + 1), sq);
        const unsigned t = __funnelshift_r(P.T.ld(wt), P.T.ld(wt + 1), st);
        const unsigned x = P.differing(q, t);
        const unsigned b = __ballot_sync(gmf::FULL_MASK, x != 0u);
        if (b) {
            const int l = __ffs((int)b) - 1;
            return i + min(at + 4 * l + ((__ffs((int)__shfl_sync(gmf::FULL_MASK, x, l)) - 1) >> 3), lim);
        }
    }
    return i + max(lim, 0);
}

// A pair is computed by one warp, or by the whole block when it is long.  A
// team keeps wavefronts beyond its shared memory as Spilled, in spill().
struct WarpTeam {
    int rank;
    int* slot;  // shared memory: the warp's slot, -1 until it needs one
    static constexpr int SIZE = 32;
    using Spilled = short;
    __device__ int top(const WfaArgs& A) const { return A.warp_eff; }
    // At most one slot per warp that computes pairs: no more than there are warps, or pairs.
    __device__ short* spill(const WfaArgs& A) const {
        if (rank == 0 && *slot < 0) *slot = (int)atomicAdd(A.warp_slots, 1u);
        __syncwarp();
        return A.warp_spill + (long long)*slot * (2 * (2 * A.warp_eff + 5));
    }
    __device__ void sync() const { __syncwarp(); }
    __device__ bool sync_any(bool x) const {
        __syncwarp();
        return __any_sync(gmf::FULL_MASK, x);
    }
    __device__ long long bcast0(long long v, long long*) const { return __shfl_sync(gmf::FULL_MASK, v, 0); }
};

template <int T>
struct BlockTeam {
    int rank;
    static constexpr int SIZE = T;
    using Spilled = int;
    __device__ int top(const WfaArgs& A) const { return A.eff; }
    __device__ int* spill(const WfaArgs& A) const {
        return A.block_spill + (long long)blockIdx.x * (2 * (2 * A.eff + 5));
    }
    __device__ void sync() const { __syncthreads(); }
    __device__ bool sync_any(bool x) const { return __syncthreads_or(x) != 0; }
    __device__ long long bcast0(long long v, long long* scratch) const {
        if (rank == 0) *scratch = v;
        __syncthreads();
        const long long r = *scratch;
        __syncthreads();
        return r;
    }
};

__device__ __forceinline__ void put_offset(int* at, int v) { *at = v; }
__device__ __forceinline__ void put_offset(short* at, int v) { *at = (short)max(v, WFA_NONE16); }

// The wavefronts of one pair up to completion; returns the distance, or -1
// once `limit` is reached without completing.  `sm` holds two wavefronts of
// scores up to `sm_s`; beyond that they move to the team's global slot (two of
// 2*top+5).
// KNOWN: `hist` is the pair's history, and only the diagonals that can still
// reach the end by `limit` (the distance) are computed.  CHUNKED: *last
// receives the offset of the last chunk, -1 when the workspace ran out.
template <Mode MODE, class Team>
__device__ int wfa_forward(const WfaArgs& A, Pair& P, int limit, int* sm, int sm_s, int* hist, long long* last,
                           const Team& tm, long long* scratch) {
    const int n = P.n, m = P.m, final_k = n - m;
    {
        bool other = false;  // (bytes around the query's ends only make the pair look less plain)
        for (int w = tm.rank; 4 * w < P.Q.shift + n; w += Team::SIZE) other |= unmatched(P.Q.ld(w)) != 0u;
        P.plain = !tm.sync_any(other);
    }
    long long h0 = 0;
    if (tm.rank < 32) h0 = wfa_extend_warp(P, 0, 0);
    h0 = tm.bcast0(h0, scratch);
    long long chunk = -1;
    int* row = nullptr;  // wavefront s is kept at row[k]
    const int own = MODE == CHUNKED ? history_share(max(n, m), limit) : 0;
    auto next_chunk = [&](int s) {  // the chunk that starts with wavefront s
        long long o = -1;
        if (tm.rank == 0) {
            o = take_chunk(A, s / WFA_CHUNK, own);
            if (o >= 0) {
                A.hist[o] = (int)(unsigned)(unsigned long long)chunk;
                A.hist[o + 1] = (int)(unsigned)((unsigned long long)chunk >> 32);
            }
        }
        chunk = tm.bcast0(o, scratch);
    };
    if (MODE == CHUNKED) {
        next_chunk(0);
        *last = chunk;
        if (tm.rank == 0 && chunk >= 0) A.hist[chunk + 2] = (int)h0;
    }
    if (MODE == KNOWN && tm.rank == 0) hist[0] = (int)h0;
    if (final_k == 0 && h0 >= n) return 0;
    // Wavefront s lies at [k + cen] with WFA_NONE two entries beyond its ends, so that every candidate can be
    // read without a look at the previous one's range.
    int cen = sm_s + 2;
    if (tm.rank < 5) sm[cen - 2 + tm.rank] = tm.rank == 2 ? (int)h0 : WFA_NONE;
    tm.sync();
    // One wavefront from the one before; true when the pair is complete.
    auto wave = [&](int s, const auto* prev, auto* cur) {
        if (MODE == CHUNKED) {
            if ((s & (WFA_CHUNK - 1)) == 0 && chunk >= 0) {
                next_chunk(s);
                *last = chunk;
            }
            row = chunk >= 0 ? A.hist + chunk + chunk_row(s) + s : nullptr;
        }
        if (MODE == KNOWN) row = hist + (long long)s * s + s;
        const int lo = MODE == KNOWN ? max(-s, final_k - (limit - s)) : -s;
        const int hi = MODE == KNOWN ? min(s, final_k + (limit - s)) : s;
        bool done = false;
        if (tm.rank < 4) put_offset(cur + cen + (tm.rank < 2 ? -s - 2 + tm.rank : s - 1 + tm.rank), WFA_NONE);
        const int lane = threadIdx.x & 31;
        for (int kw = lo + tm.rank - lane; kw <= hi; kw += Team::SIZE) {  // a warp's 32 diagonals
            const int k = kw + lane;
            const bool mine = k <= hi;
            // a candidate past the end of a sequence is none (before the start it cannot be)
            const int top = min(n, m + k);
            int sub = WFA_NONE, ins = WFA_NONE, del = WFA_NONE;
            if (mine) sub = prev[k + cen] + 1, ins = prev[k - 1 + cen] + 1, del = prev[k + 1 + cen];
            sub = sub <= top ? sub : WFA_NONE;
            ins = ins <= top ? ins : WFA_NONE;
            del = del <= top ? del : WFA_NONE;
            const int best = max(max(sub, ins), del);
            bool more = false;
            int r = best >= 0 ? wfa_extend(P, best, k, more) : WFA_NONE;
            for (unsigned b = __ballot_sync(gmf::FULL_MASK, more); b; b &= b - 1) {
                const int l = __ffs((int)b) - 1;
                const int e = wfa_extend_warp(P, __shfl_sync(gmf::FULL_MASK, r, l), kw + l);
                if (lane == l) r = e;
            }
            if (mine) {
                put_offset(cur + k + cen, r);
                if (MODE != DIST && (MODE == KNOWN || row)) row[k] = r;
                done |= (k == final_k) && r >= n;
            }
        }
        return tm.sync_any(done);
    };
    int s = 1;
    int *prev = sm, *cur = sm + 2 * sm_s + 5;
    const int top = tm.top(A);  // s <= max(n, m) <= top always holds
    for (; s <= sm_s; ++s) {
        if (s - 1 >= limit || s > top) return -1;
        if (wave(s, prev, cur)) return s;
        int* tmp = prev;
        prev = cur;
        cur = tmp;
    }
    if (s - 1 >= limit || s > top) return -1;
    // the live wavefront moves to the global slot
    typename Team::Spilled* gprev = tm.spill(A);
    typename Team::Spilled* gcur = gprev + 2 * top + 5;
    {
        const int gcen = top + 2, k0 = -(s - 1) - 2;
        for (int k = k0 + tm.rank; k <= -k0; k += Team::SIZE) put_offset(gprev + k + gcen, prev[k + cen]);
        cen = gcen;
    }
    tm.sync();
    for (;; ++s) {
        if (s - 1 >= limit || s > top) return -1;
        if (wave(s, gprev, gcur)) return s;
        auto* tmp = gprev;
        gprev = gcur;
        gcur = tmp;
    }
}

// One pair: its distance, its distance and history, or the history of its
// known distance.
template <Mode MODE, class Team>
__device__ void wfa_pair(const WfaArgs& A, int p, int* sm, int sm_s, const Team& tm, long long* scratch) {
    const long long q0 = A.q_off[p], t0 = A.t_off[p];
    const int n = (int)(A.q_off[p + 1] - q0), m = (int)(A.t_off[p + 1] - t0);
    Pair P(A.Q, q0, n, A.T, t0, m);
    if (MODE != KNOWN) {
        long long last = -1;
        const int d = n == 0 || m == 0 ? max(n, m)
                                       : wfa_forward<MODE>(A, P, A.max_distance, sm, sm_s, nullptr, &last, tm, scratch);
        if (tm.rank == 0) {
            A.distance[p] = d;
            if (MODE == CHUNKED) A.hist_off[p] = last;
        }
        return;
    }
    const int d = A.distance[p];
    long long off = -1;
    if (d > A.eff) {
        if (tm.rank == 0) atomicOr(A.err, (int)GMF_SWF_WORKSPACE);
    } else if (d >= 0 && n > 0 && m > 0) {
        const long long need = (long long)(d + 1) * (d + 1);
        if (tm.rank == 0) {
            const unsigned long long o = atomicAdd(A.hist_used, (unsigned long long)need);
            if ((long long)o + need <= A.hist_cap)
                off = (long long)o;
            else
                atomicOr(A.err, (int)GMF_SWF_WORKSPACE);
        }
        off = tm.bcast0(off, scratch);
        if (off >= 0) {
            const int got = wfa_forward<KNOWN>(A, P, d, sm, sm_s, A.hist + off, nullptr, tm, scratch);
            if (got != d) off = -1;  // cannot happen: the pass is deterministic
        }
    }
    if (tm.rank == 0) A.hist_off[p] = off;
}

template <Mode MODE>
__device__ __forceinline__ bool wfa_is_long(const WfaArgs& A, int p) {
    if (MODE == KNOWN) return A.distance[p] >= A.long_d;
    const long long n = A.q_off[p + 1] - A.q_off[p], m = A.t_off[p + 1] - A.t_off[p];
    return (n > m ? n : m) >= A.long_len;
}

// Blocks pull positions of the caller's order.  A block takes one position
// and, when its pair is long, computes it with all its warps; otherwise it
// takes positions for its other warps as well and its warps compute one pair
// each (a long pair among those goes first, block-wide).  With a longest-first
// order every long pair gets a block of its own.  It takes as many as there
// are pairs per block, so that a small batch spreads over the SMs: 500 pairs of
// 2 kb with nothing in common took 25.4 ms by 32 a block (on 16 SMs), 9.8
// ms so, 500 of 3 kb with 13% differences 3,482 and 1,624 us.
template <Mode MODE, int T>
__global__ void __launch_bounds__(T, T == WFA_WIDE ? 1 : 2) wfa_forward_kernel(WfaArgs A) {
    constexpr int WARPS = T / 32;
    extern __shared__ int s_wf[];
    __shared__ int s_pos[WARPS], s_slot[WARPS];
    __shared__ long long s_scratch;
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    if (lane == 0) s_slot[wib] = -1;
    const unsigned n = (unsigned)A.n_pairs, take = min((unsigned)WARPS, (n + gridDim.x - 1) / gridDim.x);
    for (;;) {
        if (tid == 0) {
            const unsigned first = atomicAdd(A.work, 1u);
            s_pos[0] = first < n ? (int)first : -1;
            for (int e = 1; e < WARPS; ++e) s_pos[e] = -1;
            if (first < n) {
                const int p = A.order ? A.order[first] : (int)first;
                if (!wfa_is_long<MODE>(A, p)) {
                    const unsigned more = atomicAdd(A.work, take - 1);
                    for (unsigned e = 1; e < take; ++e)
                        if (more + e - 1 < n) s_pos[e] = (int)(more + e - 1);
                }
            }
        }
        __syncthreads();
        if (s_pos[0] < 0) break;
        bool any_long = false;
        for (int e = 0; e < WARPS; ++e) {
            if (s_pos[e] < 0) continue;
            const int p = A.order ? A.order[s_pos[e]] : s_pos[e];
            if (wfa_is_long<MODE>(A, p)) {
                wfa_pair<MODE>(A, p, s_wf, block_scores(T), BlockTeam<T>{tid}, &s_scratch);
                any_long = true;
                __syncthreads();
            }
        }
        if (any_long) __syncthreads();
        if (s_pos[wib] >= 0) {
            const int p = A.order ? A.order[s_pos[wib]] : s_pos[wib];
            if (!wfa_is_long<MODE>(A, p))
                wfa_pair<MODE>(A, p, s_wf + wib * 2 * WFA_SMEM_WF, WFA_SMEM_S, WarpTeam{lane, s_slot + wib},
                               nullptr);
        }
        __syncthreads();
    }
}

struct WalkArgs {
    int n_pairs;
    const long long* q_off;
    const long long* t_off;
    const int* order;
    const int* distance;
    int* hist;                // read; a consumed wavefront's first entry then holds its step
    const long long* hist_off;
    unsigned* work;
    bool chunked;
    int* op_counts;
    uint32_t* cigar;
    long long cigar_cap;
    long long* cigar_start;
    int* cigar_len;
    unsigned long long* cigar_used;
    int* err;
};

// Walk of one pair by a warp.  The walk is a chain of dependent reads, so the
// wavefronts it can meet in its next WALK_STEPS steps are copied to shared
// memory at once: a step moves by at most one diagonal, so WALK_COLS diagonals
// around the current one hold them.  A step is then four shared loads and two
// compares; its operation and the match run before it are left in its
// wavefront's first entry.  Runs are formed from 24 or 32 steps at a time, a
// lane each: counted as the walk goes, written from the entries left behind
// once the pair's words have their place.
constexpr int WALK_STEPS = 24, WALK_COLS = 64, WALK_WARPS = 4;

// Runs of the CIGAR in back-to-front order, from steps in walk order: a run
// of matches, then one X, I or D; equal operations without matches between
// them join.
struct Runs {
    uint32_t* out;  // null while counting
    long long end;  // one past the pair's last word
    long long words;
    int open_op, open_len;  // the last operation's run, not yet counted as a word
    __device__ void init(uint32_t* o, long long e) {
        out = o;
        end = e;
        words = 0;
        open_op = -1;
        open_len = 0;
    }
    __device__ void word(long long at, int op, int len) const {
        out[end - 1 - at] = ((uint32_t)len << 4) | (uint32_t)op;
    }
    // steps 0 .. n-1, one per lane: operation 1 + b (X, I, D) after `run` matches
    __device__ void steps(int b, int run, int n, int lane) {
        const unsigned lt = (1u << lane) - 1u;
        const int up = __shfl_up_sync(gmf::FULL_MASK, b, 1);
        const bool start = lane < n && !(run == 0 && b == (lane == 0 ? open_op : up));
        const unsigned starts = __ballot_sync(gmf::FULL_MASK, start);
        const unsigned eqs = __ballot_sync(gmf::FULL_MASK, start && run > 0);
        if (!starts) {
            open_len += n;
            return;
        }
        const int first = __ffs((int)starts) - 1, last = 31 - __clz((int)starts);
        const int flush = open_len > 0 ? 1 : 0;
        if (out) {
            if (lane == 0 && flush) word(words, 1 + open_op, open_len + first);
            if (start) {
                const long long at = words + flush + __popc(starts & lt) + __popc(eqs & lt);
                if (run > 0) word(at, gmf::OP_EQ, run);
                const unsigned rest = starts & ~lt & ~(1u << lane);
                if (rest) word(at + (run > 0), 1 + b, __ffs((int)rest) - 1 - lane);
            }
        }
        words += flush + __popc(starts) - 1 + __popc(eqs);
        open_op = __shfl_sync(gmf::FULL_MASK, b, last);
        open_len = n - last;
    }
    __device__ void finish(int run, int lane) {  // the match run of wavefront 0
        if (open_len > 0) {
            if (out && lane == 0) word(words, 1 + open_op, open_len);
            ++words;
        }
        if (run > 0) {
            if (out && lane == 0) word(words, gmf::OP_EQ, run);
            ++words;
        }
    }
};

// First entry (diagonal -s) of wavefront s, from the chunk that holds it (cur)
// or the one before (before).
__device__ __forceinline__ long long history_row(const WalkArgs& A, long long cur, long long before, int c, int s) {
    if (!A.chunked) return cur + (long long)s * s;
    return ((s / WFA_CHUNK) == c ? cur : before) + chunk_row(s);
}
__device__ __forceinline__ long long chunk_link(const int* hist, long long chunk) {
    return (long long)((unsigned long long)(unsigned)hist[chunk] | (unsigned long long)(unsigned)hist[chunk + 1] << 32);
}

// The walk; counts the words and, per lane, the steps' operations (n_op: X, I,
// D) and matches.  Returns false when it meets a diagonal without a valid
// predecessor (cannot happen for a history the forward pass completed at
// distance d; checked so that a bad distance never reads outside the pair's
// history).
__device__ bool wfa_walk(const WalkArgs& A, long long off, int d, int final_k, int* tile, int lane, Runs& runs,
                         int (&n_op)[3], int& n_eq) {
    int k = final_k;
    if (k < -d || k > d) return false;
    long long cur = off;
    int c = d / WFA_CHUNK;
    const unsigned tile_at = (unsigned)__cvta_generic_to_shared(tile);
    int h0 = 0;
    for (int s = d; s >= 1;) {
        // wavefronts s .. s - WALK_STEPS, diagonals kb .. kb + WALK_COLS
        if (A.chunked)
            for (; s / WFA_CHUNK < c; --c) cur = chunk_link(A.hist, cur);
        const long long before = A.chunked && c > 0 ? chunk_link(A.hist, cur) : cur;
        const int kb = k - WALK_COLS / 2, s_hi = s, n = min(WALK_STEPS, s);
        __syncwarp();
        const int k0 = kb + lane, k1 = k0 + 32;
        for (int r = 0; r <= n; ++r) {
            const int sr = s_hi - r;
            const int* row = A.hist + history_row(A, cur, before, c, sr) + sr;
            const unsigned at = tile_at + (unsigned)(r * WALK_COLS + lane) * 4;
            if (k0 >= -sr && k0 <= sr)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(at), "l"(row + k0) : "memory");
            else
                tile[r * WALK_COLS + lane] = -1;
            if (k1 >= -sr && k1 <= sr)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(at + 128), "l"(row + k1) : "memory");
            else
                tile[r * WALK_COLS + lane + 32] = -1;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        int op = 0, run = 0;  // this lane's step
        const int* row = tile - kb;
        int reach = row[k];
        for (int u = 0; u < n; ++u) {
            row += WALK_COLS;
            const int o0 = row[k], o1 = row[k - 1], o2 = row[k + 1];
            const int v0 = o0 >= 0 ? o0 + 1 : -1, v1 = o1 >= 0 ? o1 + 1 : -1;
            int b = v1 > v0 ? 1 : 0, v = max(v0, v1);
            if (o2 > v) {
                b = 2;
                v = o2;
            }
            if (v < 0) return false;
            op = lane == u ? b : op;
            run = lane == u ? reach - v : run;
            reach = b == 0 ? o0 : (b == 1 ? o1 : o2);
            k += b == 1 ? -1 : (b == 2 ? 1 : 0);
        }
        if (lane < n) {
            A.hist[history_row(A, cur, before, c, s - lane)] = run << 2 | op;
            n_eq += run;
            n_op[0] += op == 0;
            n_op[1] += op == 1;
            n_op[2] += op == 2;
        }
        runs.steps(op, run, n, lane);
        s -= n;
        h0 = reach;
    }
    if (d == 0) h0 = A.hist[history_row(A, cur, cur, 0, 0)];
    if (lane == 0) n_eq += h0;
    runs.finish(h0, lane);
    return true;
}

// The same runs from the steps left behind.
__device__ void wfa_rewalk(const WalkArgs& A, long long off, int d, int lane, Runs& runs) {
    long long cur = off;
    int c = d / WFA_CHUNK;
    for (int s = d; s >= 1; s -= 32) {
        if (A.chunked)
            for (; s / WFA_CHUNK < c; --c) cur = chunk_link(A.hist, cur);
        const long long before = A.chunked && c > 0 ? chunk_link(A.hist, cur) : cur;
        const int n = min(32, s);
        const int x = lane < n ? A.hist[history_row(A, cur, before, c, s - lane)] : 0;
        runs.steps(x & 3, x >> 2, n, lane);
    }
    if (A.chunked)
        for (; c > 0; --c) cur = chunk_link(A.hist, cur);
    runs.finish(A.hist[history_row(A, cur, cur, 0, 0)], lane);
}

__device__ void wfa_walk_pair(const WalkArgs& A, int p, int* tile, int lane) {
    const int n = (int)(A.q_off[p + 1] - A.q_off[p]), m = (int)(A.t_off[p + 1] - A.t_off[p]);
    const int d = A.distance[p];
    const bool trivial = n == 0 || m == 0;
    const long long ho = trivial ? 0 : A.hist_off[p];
    Runs runs;
    runs.init(nullptr, 0);
    int n_op[3] = {0, 0, 0}, n_eq = 0;
    bool ok = d >= 0 && ho >= 0;
    const int miss = A.chunked && d >= 0 && ho < 0 ? -2 : -1;  // -2: a distance, but the history did not fit
    if (ok && trivial) {
        runs.words = (n > 0) + (m > 0);
        if (lane == 0) {
            n_op[1] = n;
            n_op[2] = m;
        }
    } else if (ok && !wfa_walk(A, ho, d, n - m, tile, lane, runs, n_op, n_eq)) {
        if (lane == 0) atomicOr(A.err, (int)GMF_SWF_INTERNAL);
        ok = false;
    }
    if (!ok) {
        if (lane < 4 && A.op_counts) A.op_counts[4 * p + lane] = 0;
        if (lane == 0) {
            A.cigar_start[p] = 0;
            A.cigar_len[p] = miss;
        }
        return;
    }
    const long long words = runs.words;
    n_eq = __reduce_add_sync(gmf::FULL_MASK, n_eq);
#pragma unroll
    for (int o = 0; o < 3; ++o) n_op[o] = __reduce_add_sync(gmf::FULL_MASK, n_op[o]);
    long long at = 0;
    if (lane == 0) {
        at = (long long)atomicAdd(A.cigar_used, (unsigned long long)words);
        if (A.op_counts) {
            A.op_counts[4 * p + 0] = n_eq;
            A.op_counts[4 * p + 1] = n_op[0];
            A.op_counts[4 * p + 2] = n_op[1];
            A.op_counts[4 * p + 3] = n_op[2];
        }
    }
    at = __shfl_sync(gmf::FULL_MASK, at, 0);
    if (at + words > A.cigar_cap) {
        if (lane == 0) {
            atomicOr(A.err, (int)GMF_SWF_CAPACITY);
            A.cigar_start[p] = 0;
            A.cigar_len[p] = -1;
        }
        return;
    }
    __syncwarp();
    runs.init(A.cigar, at + words);
    if (trivial) {  // the I run comes first
        if (lane == 0 && n > 0) A.cigar[at] = ((uint32_t)n << 4) | (uint32_t)gmf::OP_I;
        if (lane == 0 && m > 0) A.cigar[at + (n > 0)] = ((uint32_t)m << 4) | (uint32_t)gmf::OP_D;
    } else {
        wfa_rewalk(A, ho, d, lane, runs);
    }
    if (lane == 0) {
        A.cigar_start[p] = at;
        A.cigar_len[p] = (int)words;
    }
}

__global__ void __launch_bounds__(32 * WALK_WARPS) wfa_walk_kernel(WalkArgs A) {
    __shared__ int tiles[WALK_WARPS][(WALK_STEPS + 1) * WALK_COLS];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned nw = gridDim.x * WALK_WARPS;
    // the first pair of each warp is fixed: one warp of every block first
    for (unsigned x = wib * gridDim.x + blockIdx.x; x < (unsigned)A.n_pairs;) {
        wfa_walk_pair(A, A.order ? A.order[x] : (int)x, tiles[wib], lane);
        if (lane == 0) x = nw + atomicAdd(A.work, 1u);
        x = __shfl_sync(gmf::FULL_MASK, x, 0);
    }
}

// ---- host side ----------------------------------------------------------------
constexpr size_t ALIGN = 256;
inline size_t up(size_t x) { return (x + ALIGN - 1) & ~(ALIGN - 1); }

// Threads of a forward block: wide ones while every wavefront of a long pair
// fits a block's shared memory.
int forward_threads(int eff) { return eff <= block_scores(WFA_WIDE) ? WFA_WIDE : WFA_NARROW; }

// Persistent grid: one wide block (two heavy pairs never share an SM while
// others idle; two blocks of 512 threads took 1,839 us for the 4,000 pairs
// above) or two narrow ones per SM of a B200.  A fixed SM count keeps the workspace
// size independent of the device queried.
int grid_blocks(int n_pairs, int eff) {
    return std::max(1, std::min(n_pairs, forward_threads(eff) == WFA_WIDE ? 148 : 296));
}

// Workspace pieces: [counters | last chunks | block slots | warp slots | history]
struct Ws {
    unsigned* work;
    unsigned long long* hist_used;
    unsigned* warp_slots;
    long long* hist_off;
    int* block_spill;
    short* warp_spill;
    int* hist;
    long long hist_cap;
};

// Longest distance of a pair that one warp computes (with its distance known
// it is below WFA_LONG_D, and never leaves shared memory).
int warp_eff(int eff) { return std::min(eff, WFA_LONG_LEN - 1); }

// The pieces in order; returns the bytes before the history.
size_t place(char* p, int n_pairs, int eff, int blocks, Ws& w) {
    const size_t n = (size_t)(n_pairs > 0 ? n_pairs : 1);
    const int threads = forward_threads(eff), we = warp_eff(eff);
    const size_t warps = std::min(n, (size_t)blocks * (threads / 32));
    size_t at = 0;
    auto take = [&](size_t bytes) {
        char* q = p && bytes ? p + at : nullptr;
        at += up(bytes);
        return q;
    };
    w.work = (unsigned*)take(64);
    w.hist_used = (unsigned long long*)(w.work + 2);
    w.warp_slots = w.work + 6;
    w.hist_off = (long long*)take(sizeof(long long) * n);
    w.block_spill = (int*)take(eff > block_scores(threads) ? sizeof(int) * 2 * (2 * (size_t)eff + 5) * blocks : 0);
    w.warp_spill = (short*)take(we > WFA_SMEM_S ? sizeof(short) * 2 * (2 * (size_t)we + 5) * warps : 0);
    w.hist = (int*)(p + at);
    return at;
}

size_t fixed_bytes(int n_pairs, int eff, int blocks) {
    Ws w;
    return place(nullptr, n_pairs, eff, blocks, w);
}

int carve(void* ws, size_t bytes, int n_pairs, int eff, int blocks, Ws& w) {
    const size_t need = fixed_bytes(n_pairs, eff, blocks);
    if (!ws || bytes < need) return GMF_ERR_WORKSPACE;
    place((char*)ws, n_pairs, eff, blocks, w);
    w.hist_cap = (long long)((bytes - need) / sizeof(int));
    return GMF_OK;
}

int check_pairs(const gmf_wfa_pairs* pairs) {
    if (!pairs || pairs->n_pairs < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (pairs->n_pairs == 0) return GMF_OK;
    if (!pairs->query || !pairs->query_off || !pairs->target || !pairs->target_off) return GMF_ERR_INVALID_ARGUMENT;
    if (pairs->max_len < 0 || pairs->max_len > GMF_MAX_SEQ_LEN) return GMF_ERR_LIMIT;
    if (pairs->query_total < 0 || pairs->target_total < 0) return GMF_ERR_INVALID_ARGUMENT;
    return GMF_OK;
}

int effective(const gmf_wfa_pairs* pairs, int32_t max_distance) {
    return max_distance < pairs->max_len ? max_distance : pairs->max_len;
}

WfaArgs base_args(const gmf_wfa_pairs* pairs, int32_t max_distance, int eff, const Ws& w, long long q_total,
                  long long t_total) {
    WfaArgs a{};
    a.n_pairs = pairs->n_pairs;
    a.q_off = (const long long*)pairs->query_off;
    a.t_off = (const long long*)pairs->target_off;
    a.order = pairs->order;
    a.Q = make_seq(pairs->query, q_total);
    a.T = make_seq(pairs->target, t_total);
    a.max_distance = max_distance;
    a.eff = eff;
    a.warp_eff = warp_eff(eff);
    a.block_spill = w.block_spill;
    a.warp_spill = w.warp_spill;
    a.warp_slots = w.warp_slots;
    a.work = w.work;
    a.hist_used = w.hist_used;
    a.hist_off = w.hist_off;
    a.long_len = WFA_LONG_LEN;
    a.long_d = WFA_LONG_D;
    return a;
}

template <Mode MODE, int T>
int launch_forward_t(const WfaArgs& a, int blocks, cudaStream_t st) {
    constexpr int smem = T / 32 * 2 * WFA_SMEM_WF * (int)sizeof(int);
    GMF_CUDA_TRY(cudaFuncSetAttribute(wfa_forward_kernel<MODE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    wfa_forward_kernel<MODE, T><<<blocks, T, smem, st>>>(a);
    return gmf::cuda_status(cudaGetLastError());
}

template <Mode MODE>
int launch_forward(const WfaArgs& a, int blocks, cudaStream_t st) {
    return forward_threads(a.eff) == WFA_WIDE ? launch_forward_t<MODE, WFA_WIDE>(a, blocks, st)
                                              : launch_forward_t<MODE, WFA_NARROW>(a, blocks, st);
}

int launch_walk(const gmf_wfa_pairs* pairs, const int* distance, const gmf_wfa_results* results, const Ws& w,
                bool chunked, cudaStream_t st) {
    WalkArgs b{};
    b.n_pairs = pairs->n_pairs;
    b.q_off = (const long long*)pairs->query_off;
    b.t_off = (const long long*)pairs->target_off;
    b.order = pairs->order;
    b.distance = distance;
    b.hist = w.hist;
    b.hist_off = w.hist_off;
    b.work = w.work + 4;
    b.chunked = chunked;
    b.op_counts = results->op_counts;
    b.cigar = results->cigar;
    b.cigar_cap = results->cigar_capacity;
    b.cigar_start = (long long*)results->cigar_start;
    b.cigar_len = results->cigar_len;
    b.cigar_used = results->cigar_used;
    b.err = results->error_flags;
    const int blocks = std::min(std::max((pairs->n_pairs + WALK_WARPS - 1) / WALK_WARPS, std::min(pairs->n_pairs, 148)),
                                148 * 8);
    wfa_walk_kernel<<<blocks, 32 * WALK_WARPS, 0, st>>>(b);
    return gmf::cuda_status(cudaGetLastError());
}

int check_results(const gmf_wfa_results* r) {
    return !r || !r->cigar || !r->cigar_start || !r->cigar_len || !r->cigar_used || !r->error_flags ||
                   r->cigar_capacity < 0
               ? GMF_ERR_INVALID_ARGUMENT
               : GMF_OK;
}

}  // namespace

extern "C" size_t gmf_wfa_workspace_bytes(int32_t n_pairs, int32_t max_len, int32_t max_distance,
                                          int64_t history_entries) {
    if (n_pairs < 0 || max_len < 0 || max_distance < 0 || history_entries < 0) return 0;
    const int eff = max_distance < max_len ? max_distance : max_len;
    return fixed_bytes(n_pairs, eff, grid_blocks(n_pairs, eff)) + up(sizeof(int) * (size_t)history_entries);
}

extern "C" int64_t gmf_wfa_history_entries(int32_t n_pairs, const int32_t* query_len, const int32_t* target_len,
                                           const int32_t* distance) {
    if (n_pairs < 0 || (n_pairs > 0 && (!query_len || !target_len || !distance))) return -1;
    int64_t total = 0;
    for (int32_t p = 0; p < n_pairs; ++p) {
        if (distance[p] < 0 || query_len[p] == 0 || target_len[p] == 0) continue;
        total += (int64_t)(distance[p] + 1) * (distance[p] + 1);
    }
    return total;
}

extern "C" int gmf_wfa_distance(const gmf_wfa_pairs* pairs, int32_t max_distance, int32_t* distance,
                                void* workspace, size_t workspace_bytes, gmf_stream_t stream) {
    GMF_TRY(check_pairs(pairs));
    if (max_distance < 0 || max_distance > GMF_MAX_WFA_DISTANCE) return GMF_ERR_LIMIT;
    if (pairs->n_pairs == 0) return GMF_OK;
    if (!distance) return GMF_ERR_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    GMF_BIND_STREAM(st);
    const int eff = effective(pairs, max_distance);
    const int blocks = grid_blocks(pairs->n_pairs, eff);
    Ws w;
    GMF_TRY(carve(workspace, workspace_bytes, pairs->n_pairs, eff, blocks, w));
    WfaArgs a = base_args(pairs, max_distance, eff, w, pairs->query_total, pairs->target_total);
    a.distance = distance;
    GMF_CUDA_TRY(cudaMemsetAsync(w.work, 0, 64, st));
    return launch_forward<DIST>(a, blocks, st);
}

extern "C" int gmf_wfa_align(const gmf_wfa_pairs* pairs, const int32_t* distance, int32_t max_distance,
                             const gmf_wfa_results* results, void* workspace, size_t workspace_bytes,
                             gmf_stream_t stream) {
    GMF_TRY(check_pairs(pairs));
    if (max_distance < 0 || max_distance > GMF_MAX_WFA_DISTANCE) return GMF_ERR_LIMIT;
    if (pairs->n_pairs == 0) return GMF_OK;
    if (!distance) return GMF_ERR_INVALID_ARGUMENT;
    GMF_TRY(check_results(results));
    cudaStream_t st = (cudaStream_t)stream;
    GMF_BIND_STREAM(st);
    // the history pass replays each pair to its known distance (<= max_distance)
    const int eff = effective(pairs, max_distance);
    const int blocks = grid_blocks(pairs->n_pairs, eff);
    Ws w;
    GMF_TRY(carve(workspace, workspace_bytes, pairs->n_pairs, eff, blocks, w));
    WfaArgs a = base_args(pairs, max_distance, eff, w, pairs->query_total, pairs->target_total);
    a.distance = const_cast<int*>(distance);
    a.hist = w.hist;
    a.hist_cap = w.hist_cap;
    a.err = results->error_flags;
    GMF_CUDA_TRY(cudaMemsetAsync(w.work, 0, 64, st));
    GMF_CUDA_TRY(cudaMemsetAsync(results->error_flags, 0, sizeof(int32_t), st));
    GMF_CUDA_TRY(cudaMemsetAsync(results->cigar_used, 0, sizeof(unsigned long long), st));
    GMF_TRY(launch_forward<KNOWN>(a, blocks, st));
    return launch_walk(pairs, distance, results, w, false, st);
}

extern "C" int gmf_wfa_align_direct(const gmf_wfa_pairs* pairs, int32_t max_distance, int32_t* distance,
                                    const gmf_wfa_results* results, void* workspace, size_t workspace_bytes,
                                    gmf_stream_t stream) {
    GMF_TRY(check_pairs(pairs));
    if (max_distance < 0 || max_distance > GMF_MAX_WFA_DISTANCE) return GMF_ERR_LIMIT;
    if (pairs->n_pairs == 0) return GMF_OK;
    if (!distance) return GMF_ERR_INVALID_ARGUMENT;
    GMF_TRY(check_results(results));
    cudaStream_t st = (cudaStream_t)stream;
    GMF_BIND_STREAM(st);
    const int eff = effective(pairs, max_distance);
    const int blocks = grid_blocks(pairs->n_pairs, eff);
    Ws w;
    GMF_TRY(carve(workspace, workspace_bytes, pairs->n_pairs, eff, blocks, w));
    WfaArgs a = base_args(pairs, max_distance, eff, w, pairs->query_total, pairs->target_total);
    a.distance = distance;
    a.hist = w.hist;
    a.hist_cap = w.hist_cap;
    a.err = results->error_flags;
    GMF_CUDA_TRY(cudaMemsetAsync(w.work, 0, 64, st));
    GMF_CUDA_TRY(cudaMemsetAsync(results->error_flags, 0, sizeof(int32_t), st));
    GMF_CUDA_TRY(cudaMemsetAsync(results->cigar_used, 0, sizeof(unsigned long long), st));
    GMF_TRY(launch_forward<CHUNKED>(a, blocks, st));
    return launch_walk(pairs, distance, results, w, true, st);
}
