// Banded affine-gap Smith-Waterman with traceback, biased unsigned 16x2 form
// (sm_100a).
//
// Same recurrences and traceback decisions as the int32 form (sw32.cu, which
// restates graphmambaformer/alignment/extension.py L78-302); the cells are
// 16-bit and two of them share every 32-bit SIMD instruction.
//
// Biased cells.  Every value is stored as v + Z with Z = 4*pmax + 2 (pmax =
// the largest penalty), so the biased "-inf" N = Z - (2*pmax + 2) = 2*pmax is
// still >= 0 and every value the recurrences form stays in [pmax, smax + Z]
// with smax = match * (min(qlen, tlen) + 1).  The classifier sends a pair here
// only when smax + Z + match <= 32768 (fits_int16), so all cells are exact
// unsigned 16-bit integers, every difference that a traceback flag tests stays
// within 15 bits, and the local-alignment floor is a three-way max with Z.
// The step uses the DPX __viaddmax_u16x2 / __viaddmin_u16x2 / __vimax3_u16x2,
// byte permutes and logic on the ALU pipe, and puts its adds on the FMA pipe
// (16x2 adds of constants, multiply-adds): the ALU pipe issues at half rate
// and bounds the step.  Packed adds and subtracts never carry or borrow
// across halves.  Comparisons are differences of values known to be ordered
// (H >= M >= diag, H >= F, F >= fa, E >= ea, E >= eb), read as bit 15 of
// (difference + 0x7fff) per half.
//
// Layout: a pair is aligned by a group of L lanes (L = 8, 16 or 32, so one
// warp aligns 4, 2 or 1 pairs).  Lane k carries two "virtual lanes", 2k in the
// low halves and 2k+1 in the high halves; virtual lane v owns query rows v+1,
// v+1+2L, ... and runs two steps behind virtual lane v-1.  The low half's
// inputs from the row above come from the high half of lane k-1 through ONE
// shuffle of the packed word (H.hi, F.hi); the high half's come from the low
// half of the same lane.  A strip of 2L rows takes P = sw16_period(W, L)
// steps, a multiple of 4; the first lane of the next strip reads the last
// lane's outputs through a shared-memory delay line of D = P - 4L steps
// (a rotation of the same shuffle when D = 0).
//
// Steps run in chunks of 4, and rows always start on a chunk boundary, so
// once per chunk a lane: reads one word of target codes from a shared ring,
// reads 4 delay-line entries with one 16-byte shared-memory access (from a
// ring one chunk longer than the line, so that it never shares a slot with the
// chunk's own stores), stores one 32-bit traceback word (4 bits per cell), and
// checks the chunk's maxima for the best cell (the first maximum in
// row-then-slot order is recovered from the chunk's 4 kept H values when the
// maximum grows).
//
// Long pairs with wide bands run in the cooperative form below: the warps of
// one CTA share a pair strip by strip.

#include <stddef.h>

#include <algorithm>
#include <type_traits>

#include "sw_common.cuh"

namespace gmf {

// Traceback word of one lane and chunk, byte-planar: bit u (step u of the
// chunk) of byte h holds "H != diag" of half h, bit 4+u of byte h "F
// extends"; bit u of byte 2+h holds "H != F", bit 4+u of byte 2+h "E
// extends".  nib() turns a cell's bits into the walk's 4-bit code (H source
// 1 diagonal / 2 F / 3 E, F extends, E extends); this form stores no stop
// bit, the walk stops on the H value it tracks.
template <int L>
struct Layout16 {
    const uint32_t* bits;
    int P, W, qlen;
    __device__ uint32_t nib(int i, int d) const {
        if (d < 0 || d >= W || i < 1 || i > qlen) return 0u;
        constexpr int V = 2 * L;
        const int v = (i - 1) & (V - 1), s = (i - 1) / V;
        const long long g = (long long)s * P + 2 * v + d;
        const int k = v >> 1, h = v & 1;
        const uint32_t w = bits[(g >> 2) * L + k] >> (8 * h + (int)(g & 3));
        const uint32_t n1 = w & 1u, fc = (w >> 4) & 1u, n2 = (w >> 16) & 1u, ec = (w >> 20) & 1u;
        return (n1 ? (n2 ? 3u : 2u) : 1u) | (fc << 2) | (ec << 3);
    }
};

__device__ __forceinline__ int lo16(unsigned x) { return (int)(x & 0xFFFFu); }
__device__ __forceinline__ int hi16(unsigned x) { return (int)(x >> 16); }
__device__ __forceinline__ unsigned pack16(int lo, int hi) {
    return ((unsigned)lo & 0xFFFFu) | ((unsigned)hi << 16);
}

constexpr unsigned ONE2 = 0x00010001u;

// Unsigned 16x2 max / min(x, 1) through the DPX add-max / add-min forms,
// which issue at the full integer rate (the plain __vmaxu2 / __vminu2 do not).
__device__ __forceinline__ unsigned umax2(unsigned a, unsigned b) { return __viaddmax_u16x2(a, 0u, b); }
__device__ __forceinline__ unsigned flag2(unsigned x) { return __viaddmin_u16x2(x, 0u, ONE2); }

// Selectors building the packed target codes of one step from the chunk's
// window (bytes 0..3) and the previous chunk's last code (byte 6): low half =
// this step's code, high half = the previous step's code, zero-extended.
__device__ __forceinline__ unsigned tsel(int u) {
    return u == 0 ? 0x4640u : (u == 1 ? 0x4041u : (u == 2 ? 0x4142u : 0x4243u));
}

// ---------------------------------------------------------------------------
// The pipeline of one warp, shared by the one-warp and the cooperative
// (several warps per pair) kernels.
// ---------------------------------------------------------------------------

// The step's constants in registers: the compiler otherwise loads them from
// the parameter bank (or rebuilds them) in every chunk.
struct R16 {
    unsigned ONE, NEG1, C7;  // 1, -1, 0x7fff7fff
    unsigned MATCH2, MX, GO2, NGE2, Z2, NEG2;
    __device__ __forceinline__ explicit R16(const K16& K)
        : ONE(K.ONE), NEG1(K.NEG1), C7(0x7FFF7FFFu), MATCH2(K.MATCH2), MX(K.MX), GO2(K.GO2), NGE2(K.NGE2), Z2(K.Z2),
          NEG2(K.NEG2) {
        asm volatile("" : "+r"(ONE), "+r"(NEG1), "+r"(C7), "+r"(MATCH2), "+r"(MX), "+r"(GO2), "+r"(NGE2), "+r"(Z2),
                     "+r"(NEG2));
    }
};

// A value the compiler keeps in its register instead of rebuilding it.
__device__ __forceinline__ void keep(int& x) { asm volatile("" : "+r"(x)); }
__device__ __forceinline__ void keep(unsigned& x) { asm volatile("" : "+r"(x)); }

// Shared memory by 32-bit address.
__device__ __forceinline__ unsigned get_shared(unsigned addr) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void get_shared4(unsigned (&v)[4], unsigned addr) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void put_shared(unsigned addr, unsigned v, int pred) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p st.shared.u32 [%0], %1;\n}" ::"r"(addr), "r"(v),
                 "r"(pred) : "memory");
}

__device__ __forceinline__ void put_global(uint32_t* p, unsigned v, int pred) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p st.global.u32 [%0], %1;\n}" ::"l"(
                     __cvta_generic_to_global(p)),
                 "r"(v), "r"(pred) : "memory");
}

// Per-lane DP state carried from step to step.
struct Cells16 {
    unsigned hv, fv, hd, ml, el;  // H / F of the row above (this and the previous slot), M / E on the left
    unsigned qp;                  // query codes of the two rows (0x100 = never matches)
    unsigned acc;                 // traceback word of the chunk
};

// Four pipeline steps of one lane.  The first lane of the group takes its
// row-above inputs from rv[] (delay line or previous warp; `k0` is 0 there
// and rv[] is 0 in every other lane), the others from lane k-1 by one shuffle
// of the packed (H.hi, F.hi); lanes with `put` also store theirs at out_at.
// MASKED: half words of m[] that are 0 mark
// cells outside the band, which are reset (H = 0, M = E = F = -inf); the
// caller drops it for chunks in which no lane of the warp is at a band edge.
template <int L, bool TB, int EM, bool MASKED>
__device__ __forceinline__ void chunk16(Cells16& c, const K16& K, const R16& R, const Grp<L>& grp, int src,
                                        unsigned tw, unsigned tpv, unsigned k0, const unsigned (&rv)[4],
                                        const unsigned (&m)[4], unsigned (&hk)[4], unsigned out_at, int put) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        // Every operand half is a biased value >= pmax and every difference
        // is taken between values known to be ordered, so the adds and
        // subtracts below never carry or borrow across halves.  They are
        // written to issue on the FMA pipe: 16x2 adds of a constant, and
        // multiply-adds by the run-time constants ONE / NEG1.  The DPX
        // maxima, permutes and logic of the step all take the ALU pipe,
        // which runs at half rate and bounds the step.
        const unsigned tp = prmt(tw, tpv, tsel(u));
        const unsigned mis = flag2(c.qp ^ tp);  // 0: match, 1: mismatch
        const unsigned diag = __vadd2(c.hd, R.MATCH2) - mis * R.MX;  // one multiply-add, no borrow
        const unsigned fa = __vsub2(c.hv, R.GO2);
        unsigned F = __viaddmax_u16x2(c.fv, R.NGE2, fa);  // max(F above - ext, H above - open)
        unsigned M = __vimax3_u16x2(diag, F, R.Z2);
        const unsigned ea = __vsub2(c.ml, R.GO2);
        unsigned E = __viaddmax_u16x2(c.el, R.NGE2, ea);
        if (MASKED) {
            F = (F & m[u]) | (R.NEG2 & ~m[u]);
            M = (M & m[u]) | (R.NEG2 & ~m[u]);
            E = (E & m[u]) | (R.NEG2 & ~m[u]);
        }
        const unsigned H = MASKED ? __vimax3_u16x2(M, E, R.Z2) : umax2(M, E);  // in band H >= 0 anyway
        if (TB) {
            // Each flag is bit 15 of a half of (ordered difference + 0x7fff):
            // set when the difference is at least 1.  The classifier keeps
            // every difference within 15 bits, so the sums neither carry nor
            // borrow across halves (the 32-bit x + 0x7fff7fff may carry, and
            // the subtraction that follows takes the carry back).
            const unsigned hb = H * R.ONE + R.C7;
            const unsigned n1 = diag * R.NEG1 + hb;                // H != diag
            const unsigned n2 = F * R.NEG1 + hb;                   // H != F
            const unsigned fc = fa * R.NEG1 + (F * R.ONE + R.C7);  // F extends (F above - ext > H above - open)
            unsigned ec = 0u;                                      // E extends
            if (EM == 0) ec = ea * R.NEG1 + (E * R.ONE + R.C7);    //   open > ext: E_left - ext > M_left - open
            if (EM == 2) ec = c.el - E + K.EB2;          //   open < ext: E == E_left - ext (ties extend)
            // sign-replicated high bytes: [n1.lo n1.hi n2.lo n2.hi], [fc.lo fc.hi ec.lo ec.hi]
            const unsigned w1 = prmt(n1, n2, 0xFDB9u);
            const unsigned w2 = prmt(fc, ec, 0xFDB9u);
            const unsigned b = (w1 & (0x01010101u << u)) | (w2 & (0x10101010u << u));
            c.acc = u == 0 ? b : (c.acc | b);
        }
        const unsigned pk = prmt(H, F, 0x7632u);  // (H.hi, F.hi)
        put_shared(out_at + 4 * u, pk, put);
        const unsigned sh = grp.shfl(pk, src) * k0 + rv[u];
        c.hd = c.hv;
        c.hv = prmt(sh, H, 0x5410u);  // low: row above (lane k-1 high), high: own low
        c.fv = prmt(sh, F, 0x5432u);
        c.ml = M;
        c.el = E;
        hk[u] = H;
    }
}

// Best-cell bookkeeping, branch-free: when a half's running maximum grows,
// that half's 4 H values of the chunk and the chunk's first step are kept (a
// per-half select); the first step that reaches the final maximum is found
// once, from the kept values.  The maximum only grows on a strictly larger
// value, so the kept chunk is the one in which the final maximum first
// appears.
struct BestTrack16 {
    unsigned lb;  // running maximum per half
    unsigned sv[4];
    int g_lo, g_hi;
    __device__ __forceinline__ void init(unsigned z2) {
        lb = sv[0] = sv[1] = sv[2] = sv[3] = z2;
        g_lo = g_hi = 0;
    }
    // Run by the whole warp.  VOTE: the selects are skipped in the chunks
    // where no lane's maximum grows (with row maxima, reset at every row,
    // some lane's always does).
    template <bool VOTE>
    __device__ __forceinline__ void update(const unsigned (&hk)[4], int g0, unsigned c7) {
        const unsigned nb = __vimax3_u16x2(lb, __vimax3_u16x2(hk[0], hk[1], hk[2]), hk[3]);
        if (!VOTE || __any_sync(FULL_MASK, nb != lb)) {
            // nb >= lb in each half and the difference stays within 15 bits:
            // bit 15 of difference + 0x7fff (c7) is "grew", spread over the half
            const unsigned up = prmt(nb - lb + c7, 0u, 0xBB99u);
#pragma unroll
            for (int u = 0; u < 4; ++u) sv[u] = (hk[u] & up) | (sv[u] & ~up);
            g_lo = (up & 1u) ? g0 : g_lo;
            g_hi = (up >> 31) ? g0 : g_hi;
            lb = nb;
        }
    }
    // Steps of the first cell of each half that holds its maximum.
    __device__ __forceinline__ void positions(int& pos0, int& pos1) const {
        int u0 = 3, u1 = 3;
#pragma unroll
        for (int u = 2; u >= 0; --u) {
            if (lo16(sv[u]) == lo16(lb)) u0 = u;
            if (hi16(sv[u]) == hi16(lb)) u1 = u;
        }
        pos0 = g_lo + u0;
        pos1 = g_hi + u1;
    }
};

// (score, row, slot) ordering of the best cell: higher score, then earlier
// row, then earlier slot.
__device__ __forceinline__ bool better_cell(int oh, int oi, int od, int bh, int bi, int bd) {
    return oh > bh || (oh == bh && (oi < bi || (oi == bi && od < bd)));
}

// Progress flags between the warps of a CTA: the writer publishes with a
// release store after its ring store, the reader polls with acquire loads;
// neither waits for the thread's outstanding global loads or stores (a block
// fence would).
__device__ __forceinline__ int ld_acquire_cta(const int* p) {
    int v;
    asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v)
                 : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta(int* p, int v, int pred) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p st.release.cta.shared.b32 [%0], %1;\n}" ::"r"(
                     (unsigned)__cvta_generic_to_shared(p)),
                 "r"(v), "r"(pred) : "memory");
}

// Shared memory of one lane group: the delay line (or, cooperative, this
// warp's output ring), two copies of a ring of target codes, the band masks.
struct GroupSmem {
    uint32_t* ring;
    unsigned char* codes;
    uint4* tab;
};
__host__ __device__ inline size_t group_smem_bytes(int ring, int tring, int tabn) {
    return (size_t)ring * 4 + 2 * (size_t)tring + ((size_t)tabn + 2) * 16;
}
__device__ __forceinline__ GroupSmem group_smem(const SwArgs& a, unsigned char* base, int group) {
    GroupSmem s;
    unsigned char* p = base + (size_t)group * group_smem_bytes(a.ring, a.tring, a.tabn);
    s.ring = reinterpret_cast<uint32_t*>(p);
    s.codes = p + (size_t)a.ring * 4;
    s.tab = reinterpret_cast<uint4*>(s.codes + 2 * (size_t)a.tring);
    return s;
}

// What the cooperating warps of a CTA share (NW > 1).
struct CoopLinks {
    const uint32_t* ring_in;   // the previous warp's output ring
    int* prog;                 // per warp: ring entries published
    int* cons;                 // per warp: entries of the previous warp no longer needed
};

// Runs the strips w, w + NW, ... of one pair (NW = 1: all of them) and leaves
// the traceback words, the best cell per half (non-x-drop) or the row maxima
// (x-drop).
//
// What bounds it is the instruction count of a 4-step chunk, and with few
// pairs on the GPU the latency of its dependent steps, so everything that is
// not a cell is kept off the chunk:
//  * Target codes come from a shared ring of the codes around the band,
//    refilled 2L codes at a time (loaded one refill ahead).  Chunk starts of
//    a strip lie at multiples of 4 codes from the strip's first, except that
//    odd lanes are off by 2, so two copies of the ring (the second shifted by
//    2 codes) make every chunk one aligned word load.
//  * Codes outside the target read 0xFF, which matches nothing.  Cells left
//    of the target then compute H = 0 and E, F < 0 by themselves (E, F = 0
//    with a free gap open), which gives every cell inside the target the
//    values, and every decision a walk can take, of cells that read 0 and
//    -inf there; cells right of the target or below the query feed no cell
//    inside, and their values come from cells inside by penalties only, so
//    they never pass the best cell's score, and a cell that equals it lies in
//    a later row (or a later slot of the row).  So only the band's own edges
//    (slots < 0 and >= W) need a reset, and these are the same chunks of
//    every row: the masks of a chunk are one 16-byte load from a table.
//    With 32 lanes, chunks in which no lane starts or ends a row run without
//    masks, and the table holds only the chunks near a row's ends.  Row maxima (x-drop) must not see the cells right of the target:
//    strips that reach its end add that bound to the masks.
//  * Rows start on a counter (one compare a chunk); the next row's query
//    codes are loaded one strip ahead by all lanes at once.
// Measured on one B200 against the form that kept target words per lane in
// registers, counted every row's band per step and polled every chunk:
// instructions per 4-step chunk 190 from 284 (32 lanes, x-drop, W = 129: 180),
// 204 from 260 (8 warps); steps of a lone warp 133 cycles from 226; GCUPS on
// uniform pairs 711 from 617 (3,000 x 1,500, W = 181), 775 from 628 (888 x
// 3,000, W = 601, 4 warps), 900 from 621 (444 x 2,000, W = 3,201, 8 warps),
// 545 from 445 (20,000 x 150, W = 65, 16 lanes).
// Registers: the step needs ~110 to keep its constants and both copies of the
// chunk's values at hand.  Bounds of 95, 80 and 72 registers (20, 24 and 28
// warps an SM instead of 16) ran the same pairs at 709, 656 and 551 GCUPS
// (32 lanes) and a lone warp's steps 10, 31 and 35% slower, so the kernels ask
// for 16 warps an SM.  Pairs of 16 lanes, short and alike, take 20, which by the
// rounds that a batch makes is better or worse (us a call with 16 / 20 warps: of
// 150 bp 2,000 pairs 70 / 72, 4,700 91 / 105, 10,000 168 / 165, 20,000 299 / 313,
// 50,000 705 / 702; 20,000 of 250 bp 558 / 615, 3,000 of 1,000 bp 622 / 504).
template <int L, int NW, bool TB, bool XD, int EM>
__device__ __forceinline__ void sw16_rows(const SwArgs& a, const PairGeo& G, bool active, const Grp<L>& grp,
                                          const GroupSmem& sm, int w, int nstrips, int n_chunks, int last_chunk,
                                          uint32_t* bits, int2* rowmax, const CoopLinks& lk, BestTrack16& bt) {
    constexpr int V = 2 * L, VS = V * NW;  // rows of a strip, rows between this warp's strips
    constexpr bool COOP = NW > 1;
    // The 8-warp class (wide bands) bounds each warp's lead over the warp that
    // reads it as well: lane 31 waits until its reader has taken the entries
    // it is about to overwrite, so a ring of a.ring entries (1024) serves
    // periods up to COOP_PMAX instead of needing P + 8.  A warp's lag behind
    // its predecessor then stays within [132, a.ring + 128] steps; the lags
    // of the NW links sum to P, so with NW * 132 <= P <= NW * (a.ring + 128)
    // the warps cannot all be waiting at once.
    constexpr bool BP = NW == 8;
    const K16& K = a.k16;
    const int k = grp.k;
    const int qlen = G.qlen, tlen = G.tlen, W = G.W, P = G.P;
    const int nch = P >> 2, nE = (W - 1) >> 2;  // chunks of a period; chunk of a row's last slot (low half)
    const int c0 = G.off - G.hb;                // j = row + c0 + slot
    const int8_t* __restrict__ q = G.q;

    // ---- target codes: ring byte r of copy A is code R0 + r, of copy B code R0 + r + 2 ----
    const long long tbase = (long long)(uintptr_t)a.t & ~3ll;
    const uint32_t* __restrict__ w32 = reinterpret_cast<const uint32_t*>((uintptr_t)tbase);
    long long nw64 = 1;
    if (active) nw64 = (((long long)(uintptr_t)a.t + a.t_off[a.n_pairs] - 1 - tbase) >> 2) + 1;
    const unsigned last_word = nw64 > 0x7fffffffll ? 0x7ffffffeu : (unsigned)(nw64 - 1);
    const long long pair_t = active ? (long long)(uintptr_t)G.t - tbase : 0ll;
    int tmask = a.tring - 1;
    keep(tmask);
    const int R0 = V * w + c0;
    auto raw_codes = [&](int idx, unsigned& lo, unsigned& hi) {  // the two aligned words over codes idx .. idx+3
        if (active) {
            const int wi = (int)((pair_t + (long long)idx) >> 2);  // a negative index reads the last word
            lo = __ldg(w32 + min((unsigned)wi, last_word));
            hi = __ldg(w32 + min((unsigned)(wi + 1), last_word));
        }
    };
    auto put_codes = [&](int wd, int copy, int idx, unsigned lo, unsigned hi) {
        unsigned v = __funnelshift_r(lo, hi, (int)((pair_t + (long long)idx) & 3) * 8);
        const int below = idx < 0 ? imin(-idx, 4) : 0, above = idx + 4 > tlen ? imin(idx + 4 - tlen, 4) : 0;
        if (below) v |= below == 4 ? 0xFFFFFFFFu : (1u << (8 * below)) - 1u;
        if (above) v |= above == 4 ? 0xFFFFFFFFu : ~(0xFFFFFFFFu >> (8 * above));
        *reinterpret_cast<uint32_t*>(sm.codes + copy * a.tring + ((4 * wd) & tmask)) = v;
    };
    for (int x = k; x < 2 * nch; x += L) {  // codes of the first period, both copies
        const int wd = x >> 1, copy = x & 1, idx = R0 + 4 * wd + 2 * copy;
        unsigned lo = 0u, hi = 0u;
        raw_codes(idx, lo, hi);
        put_codes(wd, copy, idx, lo, hi);
    }
    // refills: L words (2L codes of both copies) per event, one per lane
    const int f_copy = k / (L / 2);
    int f_wd = nch + k % (L / 2);
    unsigned f_lo = 0u, f_hi = 0u;
    raw_codes(R0 + 4 * f_wd + 2 * f_copy, f_lo, f_hi);
    auto refill = [&]() {
        put_codes(f_wd, f_copy, R0 + 4 * f_wd + 2 * f_copy, f_lo, f_hi);
        f_wd += L / 2;
        raw_codes(R0 + 4 * f_wd + 2 * f_copy, f_lo, f_hi);
    };

    // ---- band masks by chunk of the row (32 lanes: chunks 0..32, then the last 33) ----
    const int n_tab = L == 32 ? imin(nch, a.tabn) : nch;
    for (int x = k; x < n_tab; x += L) {
        const int cc = x <= 32 || L < 32 ? x : x + nch - n_tab;
        unsigned mm[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = 4 * cc + u;
            mm[u] = (t <= W - 1 ? 0xFFFFu : 0u) | (t >= 2 && t <= W + 1 ? 0xFFFF0000u : 0u);
        }
        sm.tab[x] = make_uint4(mm[0], mm[1], mm[2], mm[3]);
    }
    if (k == 0) {
        const unsigned i = K.init_pk();
        sm.tab[a.tabn] = make_uint4(0u, 0u, 0u, 0u);
        sm.tab[a.tabn + 1] = make_uint4(i, i, i, i);
    }
    if (!COOP)
        for (int x = k; x < a.ring; x += L) sm.ring[x] = K.init_pk();
    __syncwarp();

    // ---- per-lane state ----
    Cells16 c;
    c.hv = c.hd = K.Z2;
    c.fv = c.ml = c.el = K.NEG2;
    c.qp = 0x01000100u;
    c.acc = 0u;
    unsigned tpv = 0u;
    bt.init(K.Z2);
    // byte offset of the lane's chunk in the mask table (n_tab entries on, the
    // next row starts; lane k's first row starts at chunk k)
    const int y_end = 16 * n_tab;
    int y = y_end - 16 * k;
    const unsigned codes_at = (unsigned)__cvta_generic_to_shared(sm.codes + (k & 1) * a.tring);
    const unsigned tab_at = (unsigned)__cvta_generic_to_shared(sm.tab);
    int pos = P - VS - 2 * k - 2 * (k & 1);  // ring byte of the chunk's codes
    // word of the chunk's traceback bits; a cooperative lane moves on to its next strip's words at the row start
    const int nch_tb = COOP ? sw16_period(W, L) >> 2 : nch;  // chunks of a strip in the words (a padded period has more)
    const int tb_jump = (NW * nch_tb - nch) * L;
    int tbi = COOP ? w * nch_tb * L - tb_jump + k : k;
    unsigned tb_lim = COOP ? 0u : (unsigned)(last_chunk + 1) * L;  // no words before a lane's first row
    const unsigned tb_all = (unsigned)(last_chunk + 1) * L;
    const int src = (k + L - 1) & (L - 1);
    const int D = P - 4 * L;  // delay-line steps, a multiple of 4 (0: a rotation of the shuffle)
    const bool from_rv = k == 0 && (COOP || D > 0);
    const int to_ring = k == L - 1 && (COOP ? !a.coop_stall : D > 0) ? 1 : 0;
    const unsigned k0 = from_rv ? 0u : 1u;
    int rmask = a.ring - 1;
    keep(rmask);
    const unsigned ring_at = (unsigned)__cvta_generic_to_shared(sm.ring);
    // The first lane reads its entries from the ring (row 0 above the first
    // strip and strips past the query: a constant entry), the others zeros.
    const unsigned const_at = (unsigned)__cvta_generic_to_shared(sm.tab + a.tabn) + (from_rv ? 16u : 0u);
    const unsigned src_at = COOP ? (unsigned)__cvta_generic_to_shared(lk.ring_in) : ring_at;
    unsigned in_at = COOP || !from_rv ? const_at : src_at;
    unsigned in_step = COOP || !from_rv ? 0u : 4u;
    int jump = VS - P;
    keep(jump);
    const R16 R(K);
    // Cooperative waits: the last progress read from the previous / next warp,
    // and how far ahead of its need a warp that has to wait lets its
    // predecessor run, so that it polls once per several chunks.  The lags of
    // the NW links sum to P, so a wait for a lag of 132 + ahead <= P / NW
    // cannot close the ring.
    int seen = 0, freed = 0;
    const int ahead = COOP ? imin(64, (P / NW - 132) & ~3) : 0;
    const int w_prev = (w + NW - 1) % NW;
    const int prev_end = COOP && w_prev < nstrips ? (((nstrips - 1 - w_prev) / NW + 1) * P + 4 * L + 4) & ~3 : 0;

    int row = V * (w - NW) + 2 * k + 1;  // the lane's low row of the current period
    unsigned nqp = 0x01000100u, nmb = 0u;
    int rq0 = row + VS <= qlen ? (int)q[row + VS - 1] : -1;
    int rq1 = row + VS + 1 <= qlen ? (int)q[row + VS] : -1;
    unsigned mb = 0u;  // x-drop: 32768 + slots inside the target per half, from the row's start
    // x-drop: the finished row's maximum, written by all lanes at once in the next period
    BestTrack16 fin;
    if (XD) fin.init(K.Z2);
    auto write_rows = [&](const BestTrack16& b, int kk) {
        const int r = V * (w + NW * kk) + 2 * k + 1;
        int p0, p1;
        b.positions(p0, p1);
        const int at = kk * P + 4 * k;
        if (active && kk >= 0) {
            if (r <= qlen) rowmax[r - 1] = make_int2((lo16(b.lb) - (int)K.Z) * K.G, p0 - at);
            if (r + 1 <= qlen) rowmax[r] = make_int2((hi16(b.lb) - (int)K.Z) * K.G, p1 - at - 2);
        }
    };

    // Polls a progress flag until it reaches `need`.  Bounded: after the
    // limit, or once any wait in the grid gave up (every later wait then ends
    // within ~1k spins), record and go on.
    auto wait_for = [&](int& have, const int* flag, int need) {
        int spins = 0;
        // the smallest of the lanes' own reads: uniform, and no lane goes on before its own read allows it
        while ((have = __reduce_min_sync(FULL_MASK, ld_acquire_cta(flag))) < need) {
            if (++spins > a.coop_spin_limit ||
                ((spins & 1023) == 0 &&
                 __any_sync(FULL_MASK, (*(volatile int*)a.err & (int)GMF_SWF_TIMEOUT) != 0))) {
                if (k == 0) atomicOr(a.err, (int)GMF_SWF_TIMEOUT);
                break;
            }
            __nanosleep(40);
        }
    };

    int kk = -1;             // the group's period (lane 0's strip)
    int next_period = 0;     // chunk at which it ends
    // Cooperative: everything that happens only every few chunks, behind one
    // compare a chunk: NW refills of 64 codes a period, one every 33 chunks (a
    // period has at least 33 * NW); waits; and, with back-pressure, the
    // reader's progress every 8 chunks.
    int limit = 0;  // chunk at which events() must run again
    int next_fill = 0x7fffffff, fills = 0;
    const int lag = 4 * L - (w == 0 ? P : 0);  // entry e = local step + lag of the previous warp
    bool reading = false;
    auto events = [&](int gc) {
        if (gc >= next_fill) {
            refill();
            next_fill = --fills > 0 ? gc + 33 : 0x7fffffff;
        }
        limit = imin(next_fill, next_period);
        if (reading) {
            const int e = 4 * gc + lag;
            if (seen < e + 4) wait_for(seen, lk.prog + w_prev, imin(e + 4 + ahead, prev_end));
            limit = imin(limit, ((seen - lag - 4) >> 2) + 1);
        }
        if (BP) {
            // the slots of steps t .. t+3 held steps t - ring .. t - ring + 3
            if (freed < 4 * gc + 4 - a.ring) wait_for(freed, lk.cons + (w + 1) % NW, 4 * gc + 4 - a.ring);
            limit = imin(limit, ((freed + a.ring - 4) >> 2) + 1);
            // the previous warp's entries before this chunk's are no longer needed (also when this strip
            // reads none)
            st_release_cta(lk.cons + w, 4 * gc + lag, k == 0 ? 1 : 0);
            limit = imin(limit, gc + 8);
        }
        limit = imax(limit, gc + 1);  // a wait that gave up
    };
    // One chunk.  MASKED: some lane may be at a band edge; SHIFT: bytes the
    // lanes move on in the mask table (0 in the middle of the rows).
    auto chunk = [&](int gc, auto masked_, auto shift_) {
        constexpr bool MASKED = decltype(masked_)::value;
        constexpr int SHIFT = decltype(shift_)::value;
        if (SHIFT && gc == next_period) {  // lane 0 of the group starts a strip
            next_period += nch;
            ++kk;
            row += VS;
            if (COOP) {
                next_fill = kk > 0 ? gc : 0x7fffffff;
                fills = NW;
                const int s0 = w + NW * kk;
                reading = s0 >= 1 && s0 < nstrips;
                if (from_rv) {
                    in_at = reading ? src_at : const_at;
                    in_step = reading ? 4u : 0u;
                }
                limit = gc;
            } else if (kk > 0) {
                refill();
            }
            nqp = pack16((rq0 >= 0 && rq0 != 5) ? rq0 : 0x100, (rq1 >= 0 && rq1 != 5) ? rq1 : 0x100);
            if (XD) {
                const int hi0 = row <= qlen ? imax(imin(W - 1, tlen - row - c0), -1) : -1;
                const int hi1 = row + 1 <= qlen ? imax(imin(W + 1, tlen - row - c0 + 1), -1) : -1;
                nmb = pack16(32768 + hi0 + 1, 32768 + hi1 + 1);
                write_rows(fin, kk - 2);
            }
            rq0 = row + VS <= qlen ? (int)q[row + VS - 1] : -1;
            rq1 = row + VS + 1 <= qlen ? (int)q[row + VS] : -1;
        }
        if (COOP && gc >= limit) events(gc);
        unsigned rv[4];
        get_shared4(rv, in_at + in_step * (unsigned)((4 * gc + (COOP ? lag : -D)) & rmask));
        if (SHIFT && y == y_end) {  // the lane starts its next row (the high half two steps later)
            y = 0;
            c.qp = nqp;
            pos += jump;
            if (COOP) {
                tbi += tb_jump;
                tb_lim = min(tb_all, (unsigned)(tbi + nch_tb * L));
            }
            if (XD) {
                mb = nmb;
                fin = bt;
                bt.lb = K.Z2;
            }
        }
        const unsigned tw = get_shared(codes_at + (unsigned)(pos & tmask));
        unsigned m[4] = {0u, 0u, 0u, 0u};
        if (MASKED) {
            get_shared4(m, tab_at + (unsigned)y);
            if (XD) {  // the slots still inside the target against the step, as bit 15 per half
#pragma unroll
                for (int u = 0; u < 4; ++u) m[u] &= prmt(mb - (unsigned)(u + 1) * ONE2, 0u, 0xBB99u);
            }
        }
        unsigned hk[4];
        chunk16<L, TB, EM, MASKED>(c, K, R, grp, src, tw, tpv, k0, rv, m, hk,
                                   ring_at + 4 * (unsigned)((4 * gc) & rmask), to_ring);
        // published before the global store, so the release does not wait on it
        if (COOP) st_release_cta(lk.prog + w, 4 * gc + 4, to_ring);
        tpv = prmt(tw, tpv, 0x4344u);  // this chunk's last code, for the next chunk's high half
        pos += 4;
        y += SHIFT;
        if (XD) mb -= 4u * ONE2;
        if (TB) {
            put_global(bits + tbi, c.acc, (L == 32 && !COOP) || (unsigned)tbi < tb_lim);
            tbi += L;
        }
        bt.template update<!XD>(hk, 4 * gc, R.C7);
        __syncwarp();
    };
    using True = std::true_type;
    using False = std::false_type;
    if (L < 32 || nE <= 32) {
        for (int gc = 0; gc < n_chunks; ++gc) chunk(gc, True{}, std::integral_constant<int, 16>{});
    } else {
        // rows start in chunks 0..31 of a period and end from chunk nE on and, in the next period, up to chunk 31
        const int y_jump = 16 * (n_tab - 32 - (nch - nE));
        int gc = 0;
        for (int base = 0;; base += nch) {
            const int e1 = imin(base + 32, n_chunks);
            for (; gc < e1; ++gc) chunk(gc, True{}, std::integral_constant<int, 16>{});
            if (gc >= n_chunks) break;
            const int e2 = imin(base + nE, n_chunks);
            // x-drop: rows that end right of the target keep the masks
            if (XD && V * (w + NW * kk + 1) + c0 + W - 1 > tlen)
                for (; gc < e2; ++gc) chunk(gc, True{}, std::integral_constant<int, 0>{});
            else
                for (; gc < e2; ++gc) chunk(gc, False{}, std::integral_constant<int, 0>{});
            y += y_jump;
        }
    }
    if (XD && n_chunks > 0) {
        // rows not yet written: the last finished one of the lanes that started a strip in the last
        // period, and the current one
        const int my = n_chunks - 1 >= k ? (n_chunks - 1 - k) / nch : -1;
        if (my == kk) write_rows(fin, kk - 1);
        write_rows(bt, my);
    }
}

// Best cell of a warp's lanes (non-x-drop): the first maximum of each half,
// from its step in the warp's schedule, as (score, row, slot).
template <int L, int NW>
__device__ __forceinline__ void lane_best16(const BestTrack16& bt, unsigned Z, int g, int k, int P, int w, int& bh,
                                            int& bi, int& bd) {
    constexpr int V = 2 * L;
    int pos0, pos1;
    bt.positions(pos0, pos1);
    const int v0 = (lo16(bt.lb) - (int)Z) * g, v1 = (hi16(bt.lb) - (int)Z) * g;  // true scores
    int r0 = 0, s0 = 0, r1 = 0, s1 = 0;
    if (v0 > 0) {
        const int tt = pos0 - 2 * (2 * k);
        const int s = tt / P;
        r0 = (w + NW * s) * V + 2 * k + 1;
        s0 = tt - s * P;
    }
    if (v1 > 0) {
        const int tt = pos1 - 2 * (2 * k + 1);
        const int s = tt / P;
        r1 = (w + NW * s) * V + 2 * k + 2;
        s1 = tt - s * P;
    }
    bh = v0;
    bi = r0;
    bd = s0;
    if (v1 > bh || (v1 == bh && v1 > 0 && (r1 < bi || (r1 == bi && s1 < bd)))) {
        bh = v1;
        bi = r1;
        bd = s1;
    }
}

// The best cell of the lanes of a group, in every lane.
template <int L>
__device__ __forceinline__ void group_best16(const Grp<L>& grp, int& bh, int& bi, int& bd) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        const int oh = grp.xr(bh, o);
        const int oi = grp.xr(bi, o);
        const int od = grp.xr(bd, o);
        if (better_cell(oh, oi, od, bh, bi, bd)) {
            bh = oh;
            bi = oi;
            bd = od;
        }
    }
}

// ---------------------------------------------------------------------------
// One group of L lanes per pair.  The traceback walk runs later, in
// sw_walk_kernel.
// ---------------------------------------------------------------------------
template <int L, bool TB, bool XD, int EM>
__device__ void sw16_group(const SwArgs& a, int p, const Grp<L>& grp, const GroupSmem& sm) {
    constexpr int V = 2 * L;
    PairGeo G = load_geo(a, p);
    const int k = grp.k;
    const bool has = p >= 0;
    const bool bad = has && (G.hb < 0 || G.hb > a.max_hb);
    bool active = has && !bad && G.qlen > 0 && G.tlen > 0;
    if (has && !active && k == 0) write_empty<TB>(a, p, bad);
    if (bad) G.W = 1;
    const int qlen = G.qlen, W = G.W;
    G.P = sw16_period(W, L);

    const unsigned long long tbw = (TB && active) ? sw16_tb_words_l(qlen, W, L) : 0ull;
    uint32_t* ws = ws_alloc<L>(a, grp, tbw + (XD && active ? 2ull * qlen : 0ull), active && (TB || XD));
    if (active && (TB || XD) && !ws) {
        if (k == 0) write_empty<TB>(a, p, true);
        active = false;
    }
    int2* rowmax = (XD && active) ? reinterpret_cast<int2*>(ws + tbw) : nullptr;
    const int nstrips = (qlen + V - 1) / V;
    const int my_last = active ? (nstrips - 1) * G.P + 2 * ((qlen - 1) % V) + W - 1 : -1;
    const int last_chunk = my_last >> 2;  // -1 when inactive
    const int n_chunks = __reduce_max_sync(FULL_MASK, last_chunk) + 1;

    BestTrack16 bt;
    sw16_rows<L, 1, TB, XD, EM>(a, G, active, grp, sm, 0, nstrips, n_chunks, last_chunk, ws, rowmax, CoopLinks{}, bt);
    __syncwarp();

    int bh, bi, bd;
    if (XD) {
        if (active && k == 0) record_rowmax(a, p, rowmax);
        xdrop_best<L>(grp, rowmax, qlen, a.x_drop, active, bh, bi, bd);
    } else {
        lane_best16<L, 1>(bt, a.k16.Z, a.k16.G, k, G.P, 0, bh, bi, bd);
        group_best16<L>(grp, bh, bi, bd);
        if (!active) bh = 0;
    }
    if (active && k == 0) {
        a.score[p] = bh;
        a.q_end[p] = bh > 0 ? bi : 0;
        a.t_end[p] = bh > 0 ? bi + G.off - G.hb + bd : 0;
        if (TB) record_walk(a, p, ws, L);
    }
}

// Warps take pairs in the list's order (longest first).  The first pair of
// each warp is fixed: pairs go to one warp of every block before a second
// one, and to different schedulers of the SM in the blocks of later waves, so
// a short list spreads over the SMs instead of filling the first blocks.
template <int L, bool TB, bool XD, int EM>
__global__ void __launch_bounds__(128, L == 16 ? 5 : 4) sw16_kernel(SwArgs a) {
    extern __shared__ uint4 sw16_smem[];
    constexpr int GPW = 32 / L;  // pairs per warp
    constexpr int CLS = L == 8 ? CLS_I16_L8 : (L == 16 ? CLS_I16_L16 : CLS_I16_L32);
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5, wpb = (int)blockDim.x >> 5;
    const int gi = lane / L;
    const GroupSmem sm = group_smem(a, reinterpret_cast<unsigned char*>(sw16_smem), wib * GPW + gi);
    Grp<L> grp(lane);
    const int count = a.queue[N_CLASSES + CLS];
    const int32_t* list = a.lists + (size_t)CLS * a.n_pairs;
    const int wave = (int)blockIdx.x / a.sms;
    int base = (((wib + wpb - wave % wpb) % wpb) * (int)gridDim.x + (int)blockIdx.x) * GPW;
    while (base < count) {
        const int idx = base + gi;
        const int p = idx < count ? list[idx] : -1;
        sw16_group<L, TB, XD, EM>(a, p, grp, sm);
        if (lane == 0) base = atomicAdd(&a.queue[CLS], GPW) + (int)gridDim.x * wpb * GPW;
        base = __shfl_sync(FULL_MASK, base, 0);
    }
}

// ---------------------------------------------------------------------------
// Cooperative form: the NW warps of one CTA align one long pair.
//
// Warp w runs strips w, w+NW, w+2NW, ... of the pair with the one-warp
// pipeline; the first lane of each strip reads the row above (the last lane's
// (H.hi, F.hi) of the strip before) from the previous warp's shared-memory
// ring instead of its own delay line.  Entry e of warp w's ring is its last
// lane's output at warp-local step e; warp w reads entry t + 4L of warp w-1
// at its local step t (t + 4L - P from warp NW-1 for warp 0), so each warp
// runs at least 4L + 4 steps behind its predecessor, and the cycle of NW
// warps keeps moving only when P >= NW * (4L + 4).  A pair with a shorter
// period than NW * a.coop_lag (4L + 4 and a little slack, so that a warp does
// not poll at every chunk) is run with this one, its lanes idle between their
// rows (at most 64 steps, or 16 chunks: the mask table covers a row's last 33).
// Under that bound no writer is ever more than P entries ahead of its reader,
// so the 2- and 4-warp classes use rings of R >= P + 8 entries and no
// back-pressure.  The 8-warp class (periods up to COOP_PMAX) adds
// back-pressure instead and keeps 1,024-entry rings: its writers also wait
// for their readers (see sw16_rows).  Each writer
// publishes its progress after every chunk (ring store, then a release store
// of the flag); each reader polls the flag with acquire loads and an
// iteration limit, after which it records GMF_SWF_TIMEOUT and goes on.
// Traceback words land at the same (strip, row step, lane) positions as in
// the one-warp layout, so the walk is unchanged.
// ---------------------------------------------------------------------------
template <int NW, bool TB, bool XD, int EM>
__device__ void sw16_coop_pair(const SwArgs& a, int p, unsigned char* smem, int* prog, int* cons, int (*sbest)[3],
                               uint32_t** sws) {
    constexpr int L = 32, V = 64;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Grp<32> grp(lane);
    PairGeo G = load_geo(a, p);
    const bool bad = G.hb < 0 || G.hb > a.max_hb;
    if (bad || G.qlen <= 0 || G.tlen <= 0) {  // uniform over the CTA
        if (threadIdx.x == 0) write_empty<TB>(a, p, bad);
        return;
    }
    const int qlen = G.qlen, W = G.W;
    G.P = imax(sw16_period(W, L), NW * a.coop_lag);
    const int P = G.P;
    const int nstrips = (qlen + V - 1) / V;
    // last chunk of the traceback words
    const int last_chunk = ((nstrips - 1) * sw16_period(W, L) + 2 * ((qlen - 1) % V) + W - 1) >> 2;

    const unsigned long long tbw = TB ? sw16_tb_words_l(qlen, W, L) : 0ull;
    if (w == 0) {
        uint32_t* ws0 = ws_alloc<32>(a, grp, tbw + (XD ? 2ull * qlen : 0ull), TB || XD);
        if (lane == 0) *sws = ws0;
    }
    if (threadIdx.x < NW) {
        prog[threadIdx.x] = 0;
        cons[threadIdx.x] = (int)threadIdx.x < nstrips ? 0 : 0x7fffffff;  // a warp without strips reads nothing
    }
    __syncthreads();
    uint32_t* ws = *sws;
    if ((TB || XD) && !ws) {
        if (threadIdx.x == 0) write_empty<TB>(a, p, true);
        return;
    }
    int2* rowmax = XD ? reinterpret_cast<int2*>(ws + tbw) : nullptr;

    const int kk_last = w < nstrips ? (nstrips - 1 - w) / NW : -1;  // this warp's last strip (local index)
    // drains what the next warp may read
    const int n_chunks = kk_last >= 0 ? ((kk_last + 1) * P + 4 * L + 4) >> 2 : 0;
    const GroupSmem sm = group_smem(a, smem, w);
    const CoopLinks lk{group_smem(a, smem, (w + NW - 1) % NW).ring, prog, cons};
    BestTrack16 bt;
    sw16_rows<L, NW, TB, XD, EM>(a, G, true, grp, sm, w, nstrips, n_chunks, last_chunk, ws, rowmax, lk, bt);
    if (NW == 8 && lane == 0 && kk_last >= 0) st_release_cta(cons + w, 0x7fffffff, 1);  // reads nothing more
    __syncthreads();  // every traceback word and row maximum is written

    int bh = 0, bi = 0, bd = 0;
    if (!XD) {
        lane_best16<L, NW>(bt, a.k16.Z, a.k16.G, lane, P, w, bh, bi, bd);
        group_best16<L>(grp, bh, bi, bd);
        if (lane == 0) {
            sbest[w][0] = bh;
            sbest[w][1] = bi;
            sbest[w][2] = bd;
        }
        __syncthreads();
    }
    if (w != 0) return;
    if (XD) {
        if (lane == 0) record_rowmax(a, p, rowmax);
        xdrop_best<L>(grp, rowmax, qlen, a.x_drop, true, bh, bi, bd);
    } else {
        bh = sbest[0][0];
        bi = sbest[0][1];
        bd = sbest[0][2];
        for (int x = 1; x < NW; ++x)
            if (better_cell(sbest[x][0], sbest[x][1], sbest[x][2], bh, bi, bd)) {
                bh = sbest[x][0];
                bi = sbest[x][1];
                bd = sbest[x][2];
            }
    }
    if (lane == 0) {
        a.score[p] = bh;
        a.q_end[p] = bh > 0 ? bi : 0;
        a.t_end[p] = bh > 0 ? bi + G.off - G.hb + bd : 0;
        if (TB) record_walk(a, p, ws, L);
    }
}

template <int NW, bool TB, bool XD, int EM>
__global__ void __launch_bounds__(32 * NW, 16 / NW) sw16_coop_kernel(SwArgs a) {
    extern __shared__ uint4 coop_smem[];
    __shared__ int prog[NW];
    __shared__ int cons[NW];
    __shared__ int sbest[NW][3];
    __shared__ uint32_t* sws;
    __shared__ int spair;
    constexpr int CLS = NW == 2 ? CLS_I16_C2 : (NW == 4 ? CLS_I16_C4 : CLS_I16_C8);
    const int count = a.queue[N_CLASSES + CLS];
    const int32_t* list = a.lists + (size_t)CLS * a.n_pairs;
    int idx = blockIdx.x;  // the first pairs go to different SMs
    while (idx < count) {
        sw16_coop_pair<NW, TB, XD, EM>(a, list[idx], reinterpret_cast<unsigned char*>(coop_smem), prog, cons, sbest,
                                       &sws);
        if (threadIdx.x == 0) spair = atomicAdd(&a.queue[CLS], 1) + (int)gridDim.x;
        __syncthreads();
        idx = spair;
        __syncthreads();
    }
}

int sw16_coop_warps(int cls) { return cls == CLS_I16_C2 ? 2 : (cls == CLS_I16_C4 ? 4 : 8); }

template <int NW, bool TB, bool XD, int EM>
static int launch_coop(const SwArgs& a, cudaStream_t stream) {
    const size_t smem = NW * group_smem_bytes(a.ring, a.tring, a.tabn);
    void (*k)(SwArgs) = sw16_coop_kernel<NW, TB, XD, EM>;
    if (smem > 48 * 1024)
        GMF_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, sms = 0, per_sm = 0;
    GMF_CUDA_TRY(cudaGetDevice(&dev));
    GMF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GMF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * NW, smem));
    if (per_sm <= 0) return GMF_ERR_LIMIT;
    k<<<sms * per_sm, 32 * NW, smem, stream>>>(a);
    return cuda_status(cudaGetLastError());
}

template <int NW, bool TB, bool XD>
static int launch_coop_e(const SwArgs& a, int e_mode, cudaStream_t s) {
    if (e_mode == 0) return launch_coop<NW, TB, XD, 0>(a, s);
    if (e_mode == 1) return launch_coop<NW, TB, XD, 1>(a, s);
    return launch_coop<NW, TB, XD, 2>(a, s);
}

template <int NW>
static int launch_coop_x(const SwArgs& a, bool tb, bool xd, int e_mode, cudaStream_t s) {
    if (tb) return xd ? launch_coop_e<NW, true, true>(a, e_mode, s) : launch_coop_e<NW, true, false>(a, e_mode, s);
    return xd ? launch_coop_e<NW, false, true>(a, e_mode, s) : launch_coop_e<NW, false, false>(a, e_mode, s);
}

int launch_sw16_coop(const SwArgs& a, int cls, bool tb, bool xd, int e_mode, cudaStream_t stream) {
    if (cls == CLS_I16_C2) return launch_coop_x<2>(a, tb, xd, e_mode, stream);
    if (cls == CLS_I16_C4) return launch_coop_x<4>(a, tb, xd, e_mode, stream);
    return launch_coop_x<8>(a, tb, xd, e_mode, stream);
}

// ---------------------------------------------------------------------------
// Deferred traceback walk of the batched form: one warp per pair, longest
// pairs first, after every DP kernel has stored its bits.
//
// A walk is a chain of dependent steps (a 20 kb ONT-like pair takes ~1,200),
// so what bounds it is the latency of one step.  The traceback words around
// the path are therefore copied to shared memory ahead of it: 32 rows at a
// time (a block), 32 slots of each row around the path's slot at the time of
// the copy, with the codes the rows and slots need, by asynchronous copies
// three blocks ahead.  Cells outside the copied slots (the path drifted) are
// read from global memory.  Per step the 32 lanes look at 32 cells of the
// diagonal (8 in a gap); matches come from one ballot, and the score of each
// lane's cell from its population count, which gives the place where the
// alignment starts.  A gap of one base is taken in the step that finds it.
// Measured on one B200 against the walk that read every cell from global
// memory and summed the scores by a shuffle scan: 64 pairs of up to 2 kb
// 189 -> 76 us, a 1,024-read serving batch (20 kb at most) 1,807 -> 673 us,
// 20,000 mixed pairs 1,977 -> 975 us, 10,000 pairs of 150 bp 37 -> 33 us.
// ---------------------------------------------------------------------------
constexpr int WALK_ROWS = 32;    // rows of a block
constexpr int WALK_SLOTS = 32;   // slots of a row in a block
constexpr int WALK_BLOCKS = 4;   // blocks held: the current one and the next three
constexpr int WALK_TWORDS = 17;  // aligned words over 63 target codes
constexpr int WALK_QWORDS = 9;   // aligned words over 32 query codes
struct WalkTile {
    uint32_t bits[WALK_BLOCKS][WALK_ROWS][9];
    uint32_t t[WALK_BLOCKS][WALK_TWORDS];
    uint32_t q[WALK_BLOCKS][WALK_QWORDS];
};

// Asynchronous 4-byte copy global -> shared, at constant byte offsets from both addresses.
template <int DST, int SRC>
__device__ __forceinline__ void copy4_async(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0+%2], [%1+%3], 4;" ::"r"(dst), "l"(src), "n"(DST), "n"(SRC) : "memory");
}
template <int X, int N, int STRIDE>
__device__ __forceinline__ void copy_row_async(unsigned dst, const void* src, int lo, int hi) {
    if constexpr (X < N) {
        if (X >= lo && X <= hi) copy4_async<4 * X, 4 * X * STRIDE>(dst, src);
        copy_row_async<X + 1, N, STRIDE>(dst, src, lo, hi);
    }
}
template <int X, int N, int STRIDE>
__device__ __forceinline__ void copy_row_async(unsigned dst, const void* src) {
    if constexpr (X < N) {
        copy4_async<4 * X, 4 * X * STRIDE>(dst, src);
        copy_row_async<X + 1, N, STRIDE>(dst, src);
    }
}

// Where both layouts keep a row's cells: slot d of row i lies at step
// step0(i) + d, SLOTS steps to a word, words STRIDE apart.
template <class Lay>
struct RowWords;
template <int L>
struct RowWords<Layout16<L>> {
    static constexpr int SHIFT = 2, STRIDE = L;
    // step0 modulo the slots of a word
    __device__ static int phase(const Layout16<L>&, int i) { return 2 * ((i - 1) & 1); }
    // the word of step0
    __device__ static const uint32_t* word0(const Layout16<L>& y, int i) {
        const int v = (i - 1) & (2 * L - 1);
        return y.bits + ((long long)((i - 1) / (2 * L)) * (y.P >> 2) + (v >> 1)) * L + (v >> 1);
    }
    // at: step modulo the slots of a word
    __device__ static bool diagonal(uint32_t w, int i, int at) { return !((w >> (8 * ((i - 1) & 1) + at)) & 1u); }
    __device__ static uint32_t nib(uint32_t w, int i, int at) {
        w >>= 8 * ((i - 1) & 1) + at;
        const uint32_t n1 = w & 1u, fc = (w >> 4) & 1u, n2 = (w >> 16) & 1u, ec = (w >> 20) & 1u;
        return (n1 ? (n2 ? 3u : 2u) : 1u) | (fc << 2) | (ec << 3);
    }
};
template <>
struct RowWords<Layout32> {
    static constexpr int SHIFT = 3, STRIDE = 32;
    __device__ static long long step0(const Layout32& y, int i) {
        return (long long)((i - 1) >> 5) * y.P + 2 * ((i - 1) & 31);
    }
    __device__ static int phase(const Layout32& y, int i) { return (int)(step0(y, i) & 7); }
    __device__ static const uint32_t* word0(const Layout32& y, int i) {
        return y.bits + (step0(y, i) >> 3) * 32 + ((i - 1) & 31);
    }
    __device__ static bool diagonal(uint32_t w, int i, int at) { return (nib(w, i, at) & 3u) == 1u; }
    __device__ static uint32_t nib(uint32_t w, int, int at) { return (w >> (at * 4)) & 15u; }
};

// Starts the copy of block b (rows 32b+1 .. 32b+32) with slots [dlo, dlo+32).
// Only words that hold a cell of the band, and code words that hold a code of
// the pair, are read.
template <class Lay>
__device__ __forceinline__ void walk_load(const Lay& lay, const PairGeo& G, unsigned tile, int b, int dlo, int lane) {
    using R = RowWords<Lay>;
    constexpr int N = (WALK_SLOTS >> R::SHIFT) + 1;
    if (b >= 0) {
        const int at = b & (WALK_BLOCKS - 1), i0 = WALK_ROWS * b;  // rows before the block
        const int i = i0 + 1 + lane;
        const int r = R::phase(lay, i);
        const int x0 = (r + dlo) >> R::SHIFT;  // word 0 of the tile's row, from the word of step0
        const uint32_t* src = R::word0(lay, i) + (long long)x0 * R::STRIDE;
        const unsigned dst = tile + (unsigned)(offsetof(WalkTile, bits) + (at * WALK_ROWS + lane) * 36);
        // words whose steps meet [step0, step0 + W)
        const int lo = -x0, hi = i <= G.qlen ? ((r + G.W - 1) >> R::SHIFT) - x0 : -1;
        if (__all_sync(FULL_MASK, lo <= 0 && hi >= N - 1))
            copy_row_async<0, N, R::STRIDE>(dst, src);
        else
            copy_row_async<0, N, R::STRIDE>(dst, src, lo, hi);
        if (lane < WALK_QWORDS) {
            const int8_t* from = G.q + i0;
            const int w = 4 * lane - (int)((uintptr_t)from & 3);  // first byte of the word, from the block's first code
            if (w < G.qlen - i0)
                copy4_async<0, 0>(tile + (unsigned)(offsetof(WalkTile, q) + (at * WALK_QWORDS + lane) * 4), from + w);
        }
        if (lane < WALK_TWORDS) {
            const int j0 = i0 + G.off - G.hb + dlo;  // index of the first row's first slot's code
            const int8_t* from = G.t + j0;
            const int w = 4 * lane - (int)((uintptr_t)from & 3);
            if (j0 + w + 4 > 0 && j0 + w < G.tlen)
                copy4_async<0, 0>(tile + (unsigned)(offsetof(WalkTile, t) + (at * WALK_TWORDS + lane) * 4), from + w);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// One cell's traceback word, from the tile where it has it.
template <class Lay>
__device__ __forceinline__ uint32_t walk_nib(const Lay& lay, const PairGeo& G, const WalkTile& T, int i, int d, int dl) {
    using R = RowWords<Lay>;
    if ((unsigned)d >= (unsigned)G.W) return 0u;
    const int r = R::phase(lay, i);
    const uint32_t w = (unsigned)(d - dl) < (unsigned)WALK_SLOTS
                           ? T.bits[((i - 1) >> 5) & (WALK_BLOCKS - 1)][(i - 1) & 31]
                                   [((r + d) >> R::SHIFT) - ((r + dl) >> R::SHIFT)]
                           : R::word0(lay, i)[(long long)((r + d) >> R::SHIFT) * R::STRIDE];
    return R::nib(w, i, (r + d) & ((1 << R::SHIFT) - 1));
}

template <class Lay>
__device__ __forceinline__ void walk_tiled(const SwArgs& a, const Lay& lay, const PairGeo& G, const WalkTile& T,
                                           int lane, int qe, int te, int score, RunWriter& rw, int& i_out,
                                           int& j_out) {
    using R = RowWords<Lay>;
    constexpr int SM = (1 << R::SHIFT) - 1;
    const unsigned tile = (unsigned)__cvta_generic_to_shared(&T);
    const bool leader = lane == 0;
    const unsigned lt = (1u << lane) - 1u;
    const int c0 = G.off - G.hb;  // j = i + c0 + slot
    const int match = a.match, mismatch = a.mismatch, hmax = 32 * match;
    int i = qe, j = te;
    int v = score;  // H of the current cell
    int B = (i - 1) >> 5;
    int dlo[WALK_BLOCKS];  // first slot of the blocks B, B - 1, B - 2, B - 3
#pragma unroll
    for (int x = 0; x < WALK_BLOCKS; ++x) {
        dlo[x] = j - i - c0 - WALK_SLOTS / 2;
        walk_load(lay, G, tile, B - x, dlo[x], lane);
    }
    bool moved = true;
    const unsigned qa = (unsigned)(uintptr_t)G.q & 3u, ta = (unsigned)((uintptr_t)G.t + (uintptr_t)(long long)c0) & 3u;
    while (i > 0 && j > 0) {
        const int d = j - i - c0;
        while (((i - 1) >> 5) < B) {
            --B;
            dlo[0] = dlo[1];
            dlo[1] = dlo[2];
            dlo[2] = dlo[3];
            dlo[3] = d - WALK_SLOTS / 2;
            walk_load(lay, G, tile, B - 3, dlo[3], lane);
            moved = true;
        }
        if (moved) {  // blocks B and B - 1 have arrived
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            __syncwarp();
            moved = false;
        }
        if ((unsigned)d >= (unsigned)G.W) break;  // outside the band: no cell to follow
        // up to 32 cells of the diagonal, one per lane
        const int nv = imin(imin(i, j), 32);
        const int ci = i - lane;
        const bool here = ((ci - 1) >> 5) == B;
        const int dl = here ? dlo[0] : dlo[1];
        const int r = R::phase(lay, ci);
        uint32_t w = 0u;
        int qc = 0, tc = 1;
        if ((unsigned)(d - dlo[0]) < (unsigned)WALK_SLOTS && (unsigned)(d - dlo[1]) < (unsigned)WALK_SLOTS) {
            const int row = (ci - 1) & 31, at = ((ci - 1) >> 5) & (WALK_BLOCKS - 1);  // (rows before 1 read other rows)
            w = T.bits[at][row][((r + d) >> R::SHIFT) - ((r + dl) >> R::SHIFT)];
            qc = reinterpret_cast<const int8_t*>(T.q[at])[qa + row];
            tc = reinterpret_cast<const int8_t*>(
                T.t[at])[((ta + (unsigned)(ci - 1 - row + dl)) & 3u) + row + (d - dl)];
        } else if (lane < nv) {
            w = R::word0(lay, ci)[(long long)((r + d) >> R::SHIFT) * R::STRIDE];
            qc = G.q[ci - 1];
            tc = G.t[j - lane - 1];
        }
        const unsigned em = __ballot_sync(FULL_MASK, codes_match((int8_t)qc, (int8_t)tc));
        bool go = lane < nv && R::diagonal(w, ci, (r + d) & SM);
        if (v <= hmax) {
            // H of the lane's cell: the carried value less the substitution scores of the cells before it
            const int ne = __popc(em & lt);
            go = go && v - ne * match + (lane - ne) * mismatch > 0;
        }
        const unsigned stop = __ballot_sync(FULL_MASK, !go);
        const int c = stop ? __ffs((int)stop) - 1 : 32;
        const unsigned cm = c < 32 ? (1u << c) - 1u : FULL_MASK;
        const unsigned mm = em & cm;
        if (mm == cm) {
            rw.add((int)OP_EQ, c, leader);
        } else {
            int pos = 0;
            while (pos < c) {  // the =/X runs of the c diagonal cells, in walk order
                const unsigned rest = mm >> pos;
                const bool eq = rest & 1u;
                int len = eq ? lead_ones<32>(rest) : (rest ? __ffs(rest) - 1 : 32);
                len = imin(len, c - pos);
                rw.add(eq ? (int)OP_EQ : (int)OP_X, len, leader);
                pos += len;
            }
        }
        i -= c;
        j -= c;
        const int ce = __popc(mm);
        v += (c - ce) * mismatch - ce * match;
        if (c == 32) continue;
        // off the matrix, or H <= 0, or no source: the alignment starts here
        if (c >= nv || v <= 0) break;
        const uint32_t wc = __shfl_sync(FULL_MASK, w, c);
        const uint32_t nb = R::nib(wc, i, (R::phase(lay, i) + d) & SM);
        if ((nb & 3u) == 0u) break;
        const bool vert = (nb & 3u) == 2u;
        const uint32_t ext = vert ? 4u : 8u;
        int n = 1;
        v += a.gap_open;
        if (nb & ext) {
            // a longer gap, 8 cells at a time: it ends with the first cell that does not extend, or at the
            // matrix edge
            n = 0;
            v -= a.gap_open;
            for (;;) {
                const int gi = vert ? i - n - lane : i, gd = vert ? d + n + lane : d - n - lane;
                const int left = (vert ? i : j) - n;
                const int bl = B - ((gi - 1) >> 5);  // block of the row, from B
                bool e = false;
                if (lane < 8 && lane < left) {
                    const int gl = bl == 0 ? dlo[0] : (bl == 1 ? dlo[1] : d + 64);  // beyond: not in the tile
                    e = (walk_nib(lay, G, T, gi, gd, bl <= 1 ? gl : gd + 1) & ext) != 0u;
                }
                const int ec = lead_ones<32>(__ballot_sync(FULL_MASK, e));  // at most 8
                v += ec * a.gap_extend;
                n += ec;
                if (ec == 8) continue;
                if (ec < left) {
                    n += 1;            // the cell that stops extending still emits its gap base
                    v += a.gap_open;   // H of the cell the gap opened from
                }
                break;
            }
        }
        rw.add(vert ? (int)OP_I : (int)OP_D, n, leader);
        if (vert)
            i -= n;
        else
            j -= n;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    i_out = i;
    j_out = j;
}

template <class Lay>
__device__ void walk_pair(const SwArgs& a, const Grp<32>& grp, int p, const PairGeo& G, WalkTile& T, const Lay& lay) {
    const int bh = a.score[p], qe = a.q_end[p], te = a.t_end[p];
    RunWriter rw;
    uint32_t* runs = ws_alloc<32>(a, grp, (unsigned long long)qe + te + 1, bh > 0);
    const bool runs_ok = bh == 0 || runs != nullptr;
    if (!runs_ok && grp.k == 0) atomicOr(a.err, (int)GMF_SWF_WORKSPACE);
    rw.init(runs);
    int qs = qe, ts = te;
    if (runs_ok && bh > 0 && qe > 0 && te > 0) walk_tiled(a, lay, G, T, grp.k, qe, te, bh, rw, qs, ts);
    finish_cigar<32>(a, grp, p, true, rw, runs_ok, qs, ts);
}

constexpr int WALK_WARPS = 4;
__global__ void __launch_bounds__(32 * WALK_WARPS) sw_walk_kernel(SwArgs a) {
    __shared__ WalkTile tiles[WALK_WARPS];
    const int lane = threadIdx.x & 31;
    WalkTile& T = tiles[threadIdx.x >> 5];
    Grp<32> grp(lane);
    const unsigned nw = gridDim.x * WALK_WARPS;
    // the first pair of each warp is fixed: one warp of every block first
    for (unsigned idx = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; idx < (unsigned)a.n_pairs;) {
        const int p = a.order ? a.order[idx] : (int)idx;
        const int tag = a.tb_tag[p];
        if (tag >= 0) {  // else no traceback: empty pair, bad band or workspace exhausted
            const PairGeo G = load_geo(a, p);
            const uint32_t* bits = a.pool + a.tb_base[p];
            if (tag == 0) {
                walk_pair(a, grp, p, G, T, Layout32{bits, imax(64, G.W + 1), G.W, G.qlen});
            } else if (tag == 8) {
                walk_pair(a, grp, p, G, T, Layout16<8>{bits, sw16_period(G.W, 8), G.W, G.qlen});
            } else if (tag == 16) {
                walk_pair(a, grp, p, G, T, Layout16<16>{bits, sw16_period(G.W, 16), G.W, G.qlen});
            } else {
                walk_pair(a, grp, p, G, T, Layout16<32>{bits, sw16_period(G.W, 32), G.W, G.qlen});
            }
        }
        if (lane == 0) idx = nw + (unsigned)atomicAdd(&a.counters[1], 1ull);
        idx = __shfl_sync(FULL_MASK, idx, 0);
    }
}

int launch_sw_walk(const SwArgs& a, cudaStream_t stream) {
    int dev = 0, sms = 0, per_sm = 0;
    GMF_CUDA_TRY(cudaGetDevice(&dev));
    GMF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GMF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sw_walk_kernel, 32 * WALK_WARPS, 0));
    const long long most = ((long long)a.n_pairs + WALK_WARPS - 1) / WALK_WARPS;  // short lists: a warp per pair
    const long long grid = std::max(most, (long long)std::min(a.n_pairs, sms));
    sw_walk_kernel<<<(int)std::min(grid, (long long)sms * (per_sm > 0 ? per_sm : 1)), 32 * WALK_WARPS, 0, stream>>>(a);
    return cuda_status(cudaGetLastError());
}

int sw16_smem_per_warp(int cls, int ring, int tring, int tabn) {
    const int L = cls == CLS_I16_L8 ? 8 : (cls == CLS_I16_L16 ? 16 : 32);
    return (32 / L) * (int)group_smem_bytes(ring, tring, tabn);
}

// A wide band's rings bound the warps an SM holds, and 4 warps a block can leave
// room that 2 or 3 would use: at half bands of 2,043 to 2,108 a warp takes 34 KB,
// so one block of 4 fits an SM, or two of 3.  The warps a block are the most
// (up to `wpb`) that keep the most resident.  1,200 pairs of 900 bp, half bands
// 2,044 / 2,080: 9,082 / 9,237 us with 4 warps a block, 6,882 / 7,001 us so.
template <int L, bool TB, bool XD, int EM>
static int launch_l(const SwArgs& a, int wpb, cudaStream_t stream) {
    const int cls = L == 8 ? CLS_I16_L8 : (L == 16 ? CLS_I16_L16 : CLS_I16_L32);
    const size_t per_warp = (size_t)sw16_smem_per_warp(cls, a.ring, a.tring, a.tabn);
    void (*k)(SwArgs) = sw16_kernel<L, TB, XD, EM>;
    if (per_warp * wpb > 48 * 1024)
        GMF_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(per_warp * wpb)));
    int dev = 0, sms = 0, per_sm = 0;  // persistent grid: every resident block of every SM
    GMF_CUDA_TRY(cudaGetDevice(&dev));
    GMF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GMF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * wpb, per_warp * wpb));
    if (per_warp > 14 * 1024) {  // (below, 16 warps fit whatever the block)
        for (int w = wpb - 1; w >= 1; --w) {
            int n = 0;
            GMF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 32 * w, per_warp * w));
            if (n * w > per_sm * wpb) {
                per_sm = n;
                wpb = w;
            }
        }
    }
    k<<<sms * (per_sm > 0 ? per_sm : 1), 32 * wpb, per_warp * wpb, stream>>>(a);
    return cuda_status(cudaGetLastError());
}

template <int L, bool TB, bool XD>
static int launch_le(const SwArgs& a, int e_mode, int wpb, cudaStream_t s) {
    if (e_mode == 0) return launch_l<L, TB, XD, 0>(a, wpb, s);
    if (e_mode == 1) return launch_l<L, TB, XD, 1>(a, wpb, s);
    return launch_l<L, TB, XD, 2>(a, wpb, s);
}

template <int L>
static int launch_lx(const SwArgs& a, bool tb, bool xd, int e_mode, int wpb, cudaStream_t s) {
    if (tb) return xd ? launch_le<L, true, true>(a, e_mode, wpb, s) : launch_le<L, true, false>(a, e_mode, wpb, s);
    return xd ? launch_le<L, false, true>(a, e_mode, wpb, s) : launch_le<L, false, false>(a, e_mode, wpb, s);
}

int launch_sw16(const SwArgs& a, int cls, bool tb, bool xd, int e_mode, int wpb,
                cudaStream_t stream) {
    if (cls == CLS_I16_L8) return launch_lx<8>(a, tb, xd, e_mode, wpb, stream);
    if (cls == CLS_I16_L16) return launch_lx<16>(a, tb, xd, e_mode, wpb, stream);
    return launch_lx<32>(a, tb, xd, e_mode, wpb, stream);
}

}  // namespace gmf
