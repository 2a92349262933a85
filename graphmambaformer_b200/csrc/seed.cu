// (w, k) minimizer seeding against a device-resident reference index.
//
// Semantics (graphmambaformer/alignment/seeding.py): pack_kmers (L105-132:
// digits = code - 1, a window holding a digit > 3 is invalid and packs to 0,
// Horner packing in int64), hash64 (L83-103: minimap2's invertible 64-bit
// hash over every packed k-mer, invalid ones included), minimizer_mask
// (L172-199: a k-mer is selected when it equals the minimum hash of at least
// one window of w consecutive k-mers, ties all kept, w clipped to the number
// of k-mers), MinimizerIndex.query (L540-545: valid & selected k-mers, in
// read order) and KmerTable.join / lookup (L257-292: every reference position
// of the key, in the table's ascending order).  The index itself (sorted
// unique keys, CSR positions, max_occ applied) is built on the host with the
// same functions and kept on the device.
//
// Layout of gmf_seed_count / gmf_seed_fill (no workspace): one CTA per
// (read, orientation).  The read (or its reverse
// complement, built on the fly) is processed in tiles of TILE k-mer
// positions: codes of the tile plus halo go to shared memory, each thread
// packs and hashes its positions, the window minima and the selection are
// computed in shared memory, and selected k-mers are looked up by binary
// search in the key table.  Pass 1 counts anchors per (read, orientation);
// pass 2 writes them at the caller's offsets, in the reference's order, with
// a block-wide scan of the per-position counts of each tile.

//
// Layout of gmf_seed_scan / gmf_seed_emit (with a workspace): see the tile
// kernel below.

#include <cub/block/block_scan.cuh>

#include "gmf_common.cuh"

namespace {

constexpr int SEED_THREADS = 256;
constexpr int SEED_TILE = 1024;   // k-mer positions per tile
constexpr int SEED_MAX_K = 31;
constexpr int SEED_MAX_W = 256;

__device__ __forceinline__ unsigned long long mm_hash64(unsigned long long x) {
    x = (~x) + (x << 21);
    x ^= x >> 24;
    x = x + (x << 3) + (x << 8);
    x ^= x >> 14;
    x = x + (x << 2) + (x << 4);
    x ^= x >> 28;
    x = x + (x << 31);
    return x;
}

__device__ __forceinline__ int8_t seq_code(const int8_t* read, int L, int rc, int x) {
    if (!rc) return read[x];
    const int8_t c = read[L - 1 - x];
    return (c >= 1 && c <= 4) ? (int8_t)(5 - c) : c;  // reverse_complement_codes
}

struct SeedArgs {
    int k, w;
    long long n_keys;
    const long long* keys;
    const long long* offsets;
    const int32_t* positions;
    int n_reads;
    const int8_t* codes;
    const long long* read_off;
    int both;
    long long* counts;         // pass 1: 2 per read
    const long long* aoff;     // pass 2: 2 * n_reads + 1
    int32_t* read_pos;
    int32_t* ref_pos;
    int32_t* length;
    int8_t* strand;
};

// First index with keys[i] >= x.
__device__ __forceinline__ long long lower_bound(const long long* keys, long long n, long long x) {
    long long lo = 0, hi = n;
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (__ldg(keys + mid) < x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

template <bool FILL>
__global__ void __launch_bounds__(SEED_THREADS) seed_kernel(SeedArgs a) {
    using Scan = cub::BlockScan<long long, SEED_THREADS>;
    __shared__ typename Scan::TempStorage scan_tmp;
    __shared__ int8_t s_code[SEED_TILE + 2 * SEED_MAX_W + SEED_MAX_K];
    __shared__ unsigned long long s_hash[SEED_TILE + 2 * SEED_MAX_W];
    __shared__ long long s_pack[SEED_TILE];
    __shared__ unsigned char s_valid[SEED_TILE];
    __shared__ unsigned long long s_wmin[SEED_TILE + SEED_MAX_W];
    __shared__ long long s_total;
    constexpr int PER = SEED_TILE / SEED_THREADS;

    const int k = a.k;
    for (int seg = blockIdx.x; seg < 2 * a.n_reads; seg += gridDim.x) {
        const int r = seg >> 1, rc = seg & 1;
        if (rc && !a.both) {
            if (!FILL && threadIdx.x == 0) a.counts[seg] = 0;
            continue;
        }
        const long long r0 = a.read_off[r];
        const int L = (int)(a.read_off[r + 1] - r0);
        const int8_t* read = a.codes + r0;
        const int m = L - k + 1;  // k-mer positions
        if (threadIdx.x == 0) s_total = 0;
        __syncthreads();
        if (m > 0) {
            const int ww = a.w < 1 ? 1 : (a.w < m ? a.w : m);
            const int n_win = m - ww + 1;
            long long out_base = FILL ? a.aoff[seg] : 0;
            for (int t0 = 0; t0 < m; t0 += SEED_TILE) {
                // hashed positions [h0, h1): windows starting in [t0 - ww + 1, t0 + TILE) and their k-mers
                const int h0 = t0 - ww + 1 > 0 ? t0 - ww + 1 : 0;
                const int h1 = t0 + SEED_TILE + ww - 1 < m ? t0 + SEED_TILE + ww - 1 : m;
                const int c1 = h1 + k - 1;  // codes [h0, c1)
                for (int x = threadIdx.x; x < c1 - h0; x += SEED_THREADS) s_code[x] = seq_code(read, L, rc, h0 + x);
                __syncthreads();
                for (int x = threadIdx.x; x < h1 - h0; x += SEED_THREADS) {
                    long long packed = 0;
                    bool bad = false;
                    for (int o = 0; o < k; ++o) {
                        const long long dg = (long long)s_code[x + o] - 1;
                        bad |= dg > 3;
                        packed = packed * 4 + dg;
                    }
                    if (bad) packed = 0;
                    s_hash[x] = mm_hash64((unsigned long long)packed);
                    const int p = h0 + x;
                    if (p >= t0 && p < t0 + SEED_TILE) {
                        s_pack[p - t0] = packed;
                        s_valid[p - t0] = bad ? 0 : 1;
                    }
                }
                __syncthreads();
                // window minima for windows j in [jw0, jw1)
                const int jw0 = h0, jw1 = (t0 + SEED_TILE < n_win) ? t0 + SEED_TILE : n_win;
                for (int j = jw0 + threadIdx.x; j < jw1; j += SEED_THREADS) {
                    unsigned long long mn = s_hash[j - h0];
                    for (int o = 1; o < ww; ++o) {
                        const unsigned long long v = s_hash[j - h0 + o];
                        mn = v < mn ? v : mn;
                    }
                    s_wmin[j - jw0] = mn;
                }
                __syncthreads();
                // per position: selected & valid -> key lookup -> anchor count
                long long cnt[PER];
                long long kfirst[PER];
#pragma unroll
                for (int e = 0; e < PER; ++e) {
                    const int i = t0 + threadIdx.x * PER + e;
                    cnt[e] = 0;
                    kfirst[e] = 0;
                    if (i < m && s_valid[i - t0]) {
                        const unsigned long long h = s_hash[i - h0];
                        const int jlo = i - ww + 1 > 0 ? i - ww + 1 : 0;
                        const int jhi = i < n_win - 1 ? i : n_win - 1;
                        bool sel = false;
                        for (int j = jlo; j <= jhi && !sel; ++j) sel = s_wmin[j - jw0] == h;
                        if (sel) {
                            const long long key = s_pack[i - t0];
                            const long long at = lower_bound(a.keys, a.n_keys, key);
                            if (at < a.n_keys && __ldg(a.keys + at) == key) {
                                kfirst[e] = __ldg(a.offsets + at);
                                cnt[e] = __ldg(a.offsets + at + 1) - kfirst[e];
                            }
                        }
                    }
                }
                long long excl[PER];
                long long tile_total = 0;
                Scan(scan_tmp).ExclusiveSum(cnt, excl, tile_total);
                if (FILL) {
                    const int8_t sgn = rc ? (int8_t)-1 : (int8_t)1;
#pragma unroll
                    for (int e = 0; e < PER; ++e) {
                        const int i = t0 + threadIdx.x * PER + e;
                        for (long long c = 0; c < cnt[e]; ++c) {
                            const long long o = out_base + excl[e] + c;
                            a.read_pos[o] = i;
                            a.ref_pos[o] = __ldg(a.positions + kfirst[e] + c);
                            a.length[o] = k;
                            a.strand[o] = sgn;
                        }
                    }
                    out_base += tile_total;
                } else if (threadIdx.x == 0) {
                    s_total += tile_total;
                }
                __syncthreads();
            }
        }
        if (!FILL && threadIdx.x == 0) a.counts[seg] = s_total;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Scan and emit with a workspace.
//
// The forms above walk a read tile by tile in one CTA, once to count and once
// to fill, with a 21-step binary search per selected k-mer: 27 us a tile, so
// a batch took as long as its longest read (20 kb: 541 us, twice).  Here
// every tile of TILE k-mer positions is a block's work of its own, so the
// batch spreads over the SMs; a block packs and hashes both orientations of
// its k-mers (the reverse complement's k-mer at position m-1-i covers the
// same bases as the forward one at i, and its windows the same positions),
// takes the window minima by doubling (log2 w rounds on pairs of hashes), and
// looks the selected k-mers up in the index once, through a prefix table (one
// load instead of ~20 dependent ones).  The selected positions and their keys
// stay in the workspace; the emit pass only expands them.
// What bounds it now is the hash and minimum arithmetic (about 280
// instructions a position, 600 with the k-mers packed base by base) and, for
// small batches, the four launches.  Measured on one B200, 1,024 reads of
// 150-20,000 bases on a 1.2 Mb reference: 110 us + 22 us (emit) against
// 541 + 543 us.
// ---------------------------------------------------------------------------
constexpr int TILE = 512;
constexpr int TILE_THREADS = 256;
constexpr int TILE_HASHES = TILE + 2 * (SEED_MAX_W - 1);

struct TileArgs {
    SeedArgs s;
    int bits;               // prefix table (0: none)
    const int32_t* first;
    long long total;        // codes that may be read
    long long slots;        // tile slots the workspace holds
    int32_t* n_sel;         // per slot: selected k-mers, forward and reverse
    long long* n_anchor;    // per slot: anchors, forward and reverse
    int32_t* at;            // per slot: key index (-1: no hit) of each selected k-mer, forward then reverse
    unsigned short* pos;    // per slot: its position in the tile, forward then reverse
    long long* counts;      // per (read, orientation): anchors
    const long long* off;   // emit: anchor offsets
};

// A read's first code.  The workspace holds the slots of `total` codes, so a
// read that goes on beyond them is cut there.
__device__ __forceinline__ long long tile_off(const TileArgs& a, int r) {
    const long long o = a.s.read_off[r];
    return o < a.total ? o : a.total;
}

// Read r owns the tile slots from (its offset) / TILE + r on: at least as many
// as it has tiles, and never more than total / TILE + n_reads in all.
__device__ __forceinline__ long long first_slot(const TileArgs& a, int r) {
    return (tile_off(a, r) - tile_off(a, 0)) / TILE + r;
}

// The read of a slot: the last r with first_slot(r) <= slot.  32 reads are
// compared at a time by a warp.
__device__ __forceinline__ int slot_read(const TileArgs& a, long long slot, int lane) {
    int lo = 0, n = a.s.n_reads;  // the read lies in [lo, lo + n)
    while (n > 1) {
        const int step = (n + 31) / 32;
        const int r = lo + lane * step;
        const bool le = lane * step < n && first_slot(a, r) <= slot;
        const unsigned b = __ballot_sync(gmf::FULL_MASK, le);
        const int k = 31 - __clz((int)b);  // lane 0 always is
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

// Slots the batch fills (the workspace may hold more).
__device__ __forceinline__ long long used_slots(const TileArgs& a) {
    const long long n = first_slot(a, a.s.n_reads);
    return n < a.slots ? n : a.slots;
}

__device__ __forceinline__ long long find_key(const TileArgs& a, long long key) {
    long long lo = 0, hi = a.s.n_keys;
    if (a.bits > 0 && key >= 0 && (key >> (2 * a.s.k)) == 0) {
        const long long b = key >> (2 * a.s.k - a.bits);
        lo = __ldg(a.first + b);
        hi = __ldg(a.first + b + 1);
    }
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        const long long v = __ldg(a.s.keys + mid);
        if (v == key) return mid;
        if (v < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return -1;
}

// The packed k-mers at base x of a tile whose codes are all A, C, G or T:
// forward from words that hold the first base in their top bits, reverse
// complement from words of complemented digits with the first base in their
// low bits.
constexpr int TILE_WORDS = (TILE_HASHES + SEED_MAX_K) / 16 + 4;
__device__ __forceinline__ ulonglong2 kmer_pair(const uint32_t* fw, const uint32_t* rc, int x, int k) {
    const int w = x >> 4, sh = 2 * (x & 15);
    const uint32_t a0 = __funnelshift_l(fw[w + 1], fw[w], sh), a1 = __funnelshift_l(fw[w + 2], fw[w + 1], sh);
    const uint32_t b0 = __funnelshift_r(rc[w], rc[w + 1], sh), b1 = __funnelshift_r(rc[w + 1], rc[w + 2], sh);
    return make_ulonglong2(((unsigned long long)a0 << 32 | a1) >> (64 - 2 * k),
                           ((unsigned long long)b1 << 32 | b0) & ((1ull << (2 * k)) - 1ull));
}

// The same for any codes (1..4 are A, C, G, T; a digit above 3 makes the k-mer
// invalid, packed to 0).
__device__ __forceinline__ ulonglong2 kmer_pair_any(const int8_t* code, int k, bool& bad) {
    unsigned long long f = 0, c = 0;
    bad = false;
    for (int o = 0; o < k; ++o) {
        const int dg = (int)code[o] - 1;
        bad |= dg > 3;
        f = f * 4 + (unsigned long long)(long long)dg;
        // reverse_complement_codes: 1..4 -> 4..1, others kept
        const int dc = (unsigned)dg < 4u ? 3 - dg : dg;
        c += (unsigned long long)(long long)dc << (2 * o);
    }
    return bad ? make_ulonglong2(0ull, 0ull) : make_ulonglong2(f, c);
}

__global__ void __launch_bounds__(TILE_THREADS) seed_tile_kernel(TileArgs a) {
    __shared__ ulonglong2 s_a[TILE_HASHES], s_b[TILE_HASHES];  // (forward, reverse) hashes, minima, maxima
    __shared__ ulonglong2 s_hash[TILE];                        // the tile's own hashes
    __shared__ uint32_t s_fw[TILE_WORDS], s_rc[TILE_WORDS];    // digits, 16 to a word (see kmer_pair)
    __shared__ int8_t s_code[TILE_HASHES + SEED_MAX_K];
    __shared__ bool s_valid[TILE];
    __shared__ unsigned short s_pos[2 * TILE];
    __shared__ int s_cnt[2][TILE / 32], s_read;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int k = a.s.k, both = a.s.both;
    const long long n_slots = used_slots(a);
    for (long long slot = blockIdx.x; slot < n_slots; slot += gridDim.x) {
        __syncthreads();
        if (wid == 0) {
            const int r = slot_read(a, slot, lane);
            if (lane == 0) s_read = r;
        }
        __syncthreads();
        const int r = s_read;
        const long long r0 = tile_off(a, r);
        const int L = (int)(tile_off(a, r + 1) - r0);
        const int m = L - k + 1;  // k-mer positions
        const long long t0l = (slot - first_slot(a, r)) * TILE;
        if (t0l >= m) {  // a slot beyond the read's tiles (or past the last read)
            if (tid < 2) {
                a.n_sel[2 * slot + tid] = 0;
                a.n_anchor[2 * slot + tid] = 0;
            }
            continue;
        }
        const int t0 = (int)t0l, t1 = min(t0 + TILE, m);
        const int ww = a.s.w < 1 ? 1 : (a.s.w < m ? a.s.w : m);
        const int n_win = m - ww + 1;
        // hashed positions [h0, h1): the windows that cover the tile
        const int h0 = max(t0 - ww + 1, 0), h1 = min(t1 + ww - 1, m), H = h1 - h0;
        bool other = false;
        for (int x = tid; x < H + k - 1; x += TILE_THREADS) {
            const int8_t c = a.s.codes[r0 + h0 + x];
            s_code[x] = c;
            other |= c < 1 || c > 4;
        }
        const bool plain = !__syncthreads_or(other);
        if (plain) {
            for (int x = tid; x < (H + k - 1 + 15) / 16 + 2; x += TILE_THREADS) {
                uint32_t f = 0, c = 0;
                for (int o = 0; o < 16; ++o) {
                    const uint32_t dg = 16 * x + o < H + k - 1 ? (uint32_t)(s_code[16 * x + o] - 1) : 0u;
                    f |= dg << (30 - 2 * o);
                    c |= (3u - dg) << (2 * o);
                }
                s_fw[x] = f;
                s_rc[x] = c;
            }
            __syncthreads();
        }
        for (int x = tid; x < H; x += TILE_THREADS) {
            bool bad = false;
            const ulonglong2 key = plain ? kmer_pair(s_fw, s_rc, x, k) : kmer_pair_any(s_code + x, k, bad);
            const ulonglong2 h = make_ulonglong2(mm_hash64(key.x), mm_hash64(key.y));
            s_a[x] = h;
            const int p = h0 + x;
            if (p >= t0 && p < t1) {
                s_hash[p - t0] = h;
                s_valid[p - t0] = !bad;
            }
        }
        __syncthreads();
        // window minima by doubling: after a round of span s, x holds the minimum of [x, x + s)
        ulonglong2 *src = s_a, *dst = s_b;
        int span = 1;
        while (span < ww) {
            const int sh = min(span, ww - span);
            for (int x = tid; x < H; x += TILE_THREADS) {
                ulonglong2 v = src[x];
                if (x + sh < H) {
                    const ulonglong2 u = src[x + sh];
                    v.x = min(v.x, u.x);
                    v.y = min(v.y, u.y);
                }
                dst[x] = v;
            }
            __syncthreads();
            ulonglong2* t = src;
            src = dst;
            dst = t;
            span += sh;
        }
        // windows [h0, ..) hold their minimum at their first position; windows past the last one hold 0.
        // A k-mer is selected when the largest minimum of the windows that cover it, [i - ww + 1, i], is its
        // own hash (no window's minimum exceeds it).
        for (int x = tid; x < H; x += TILE_THREADS)
            if (h0 + x >= n_win) src[x] = make_ulonglong2(0ull, 0ull);
        __syncthreads();
        span = 1;
        while (span < ww) {
            const int sh = min(span, ww - span);
            for (int x = tid; x < H; x += TILE_THREADS) {
                ulonglong2 v = src[x];
                if (x >= sh) {
                    const ulonglong2 u = src[x - sh];
                    v.x = max(v.x, u.x);
                    v.y = max(v.y, u.y);
                }
                dst[x] = v;
            }
            __syncthreads();
            ulonglong2* t = src;
            src = dst;
            dst = t;
            span += sh;
        }
        // selected positions, in order: counts per 32 positions, then places
        unsigned bal[2][TILE / TILE_THREADS];
#pragma unroll
        for (int e = 0; e < TILE / TILE_THREADS; ++e) {
            const int x = e * TILE_THREADS + tid;
            bool sf = false, sr = false;
            if (t0 + x < t1) {
                if (s_valid[x]) {
                    const ulonglong2 mx = src[t0 + x - h0], h = s_hash[x];
                    sf = mx.x == h.x;
                    sr = both && mx.y == h.y;
                }
            }
            bal[0][e] = __ballot_sync(gmf::FULL_MASK, sf);
            bal[1][e] = __ballot_sync(gmf::FULL_MASK, sr);
            if (lane == 0) {
                s_cnt[0][e * (TILE_THREADS / 32) + wid] = __popc(bal[0][e]);
                s_cnt[1][e * (TILE_THREADS / 32) + wid] = __popc(bal[1][e]);
            }
        }
        __syncthreads();
        if (wid < 2 && lane < TILE / 32) {  // exclusive scan of the 16 counts of each orientation
            const int v = s_cnt[wid][lane];
            int incl = v;
#pragma unroll
            for (int o = 1; o < TILE / 32; o <<= 1) {
                const int u = __shfl_up_sync((1u << (TILE / 32)) - 1u, incl, o);
                if (lane >= o) incl += u;
            }
            s_cnt[wid][lane] = incl - v;
            if (lane == TILE / 32 - 1) a.n_sel[2 * slot + wid] = incl;
        }
        __syncthreads();
        int n_all[2];
#pragma unroll
        for (int o = 0; o < 2; ++o)
#pragma unroll
            for (int e = 0; e < TILE / TILE_THREADS; ++e) {
                const int at = s_cnt[o][e * (TILE_THREADS / 32) + wid] + __popc(bal[o][e] & ((1u << lane) - 1u));
                if ((bal[o][e] >> lane) & 1u) s_pos[o * TILE + at] = (unsigned short)(e * TILE_THREADS + tid);
            }
        __syncthreads();
        n_all[0] = a.n_sel[2 * slot];
        n_all[1] = a.n_sel[2 * slot + 1];
        // lookups, one per thread; the anchor counts per orientation
        const int total = n_all[0] + n_all[1];
        long long cnt[2] = {0, 0};
        for (int x = tid; x < total; x += TILE_THREADS) {
            const int o = x < n_all[0] ? 0 : 1;
            const int n = o ? x - n_all[0] : x;
            const int p = s_pos[o * TILE + n];
            bool bad;
            const ulonglong2 key =
                plain ? kmer_pair(s_fw, s_rc, t0 + p - h0, k) : kmer_pair_any(s_code + (t0 + p - h0), k, bad);
            const long long at = find_key(a, (long long)(o ? key.y : key.x));
            const long long slot_o = (2 * slot + o) * TILE + n;
            a.pos[slot_o] = (unsigned short)p;
            a.at[slot_o] = (int32_t)at;
            if (at >= 0) cnt[o] += __ldg(a.s.offsets + at + 1) - __ldg(a.s.offsets + at);
        }
#pragma unroll
        for (int o = 0; o < 2; ++o) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) cnt[o] += __shfl_xor_sync(gmf::FULL_MASK, cnt[o], d);
        }
        __shared__ long long s_sum[2][TILE_THREADS / 32];
        if (lane == 0) {
            s_sum[0][wid] = cnt[0];
            s_sum[1][wid] = cnt[1];
        }
        __syncthreads();
        if (tid < 2) {
            long long n = 0;
            for (int x = 0; x < TILE_THREADS / 32; ++x) n += s_sum[tid][x];
            a.n_anchor[2 * slot + tid] = n;
            if (n) atomicAdd((unsigned long long*)&a.counts[2 * r + tid], (unsigned long long)n);
        }
    }
}

// Offsets of the reads' anchors from their counts, their total and the
// largest read's: one block.
__global__ void __launch_bounds__(1024) seed_offsets_kernel(int n_reads, const long long* counts, long long* off,
                                                            long long* totals, long long* read_off) {
    using Scan = cub::BlockScan<long long, 1024>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ long long s_max[32];
    long long base = 0, most = 0;
    for (int r0 = 0; r0 < n_reads; r0 += 1024) {
        const int r = r0 + (int)threadIdx.x;
        const long long f = r < n_reads ? counts[2 * r] : 0, c = r < n_reads ? counts[2 * r + 1] : 0;
        long long excl = 0, sum = 0;
        Scan(tmp).ExclusiveSum(f + c, excl, sum);
        if (r < n_reads) {
            off[2 * r] = base + excl;
            off[2 * r + 1] = base + excl + f;
            if (read_off) read_off[r] = base + excl;
        }
        most = max(most, f + c);
        base += sum;
        __syncthreads();
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) most = max(most, __shfl_xor_sync(gmf::FULL_MASK, most, d));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = most;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int x = 1; x < 32; ++x) most = max(most, s_max[x]);
        off[2 * n_reads] = base;
        if (read_off) read_off[n_reads] = base;
        totals[0] = base;
        totals[1] = most;
    }
}

// One block per tile slot and orientation: the anchors of the slot's selected
// k-mers.  The reverse complement's anchors come in its own read order, from
// the last tile's last k-mer down.
__global__ void __launch_bounds__(128) seed_emit_kernel(TileArgs a) {
    using Scan = cub::BlockScan<long long, 128>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int s_read;
    __shared__ long long s_sum[4];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const long long n_slots = used_slots(a);
    for (long long x = blockIdx.x; x < 2 * n_slots; x += gridDim.x) {
        const long long slot = x >> 1;
        const int o = (int)(x & 1);
        const int n = a.n_sel[x];
        if (n == 0 || a.n_anchor[x] == 0) continue;  // uniform over the block
        __syncthreads();
        if (wid == 0) {
            const int r = slot_read(a, slot, lane);
            if (lane == 0) s_read = r;
        }
        __syncthreads();
        const int r = s_read;
        const int m = (int)(tile_off(a, r + 1) - tile_off(a, r)) - a.s.k + 1;
        const long long first = first_slot(a, r), last = first + (m - 1) / TILE;
        // anchors of the read's tiles before this one, in the orientation's order
        long long before = 0;
        const long long s0 = o ? slot + 1 : first, s1 = o ? last + 1 : slot;
        for (long long s = s0 + tid; s < s1; s += 128) before += a.n_anchor[2 * s + o];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(gmf::FULL_MASK, before, d);
        if (lane == 0) s_sum[wid] = before;
        __syncthreads();
        long long base = a.off[2 * r + o] + s_sum[0] + s_sum[1] + s_sum[2] + s_sum[3];
        const int t0 = (int)(slot - first) * TILE;
        for (int e0 = 0; e0 < n; e0 += 128) {
            const int e = e0 + tid;
            long long cnt = 0, key0 = 0;
            int p = 0;
            if (e < n) {
                const long long at = x * TILE + (o ? n - 1 - e : e);
                p = t0 + (int)a.pos[at];
                const int32_t key = a.at[at];
                if (key >= 0) {
                    key0 = __ldg(a.s.offsets + key);
                    cnt = __ldg(a.s.offsets + key + 1) - key0;
                }
            }
            long long excl = 0, sum = 0;
            Scan(tmp).ExclusiveSum(cnt, excl, sum);
            for (long long c = 0; c < cnt; ++c) {
                const long long w = base + excl + c;
                a.s.read_pos[w] = o ? m - 1 - p : p;
                a.s.ref_pos[w] = __ldg(a.s.positions + key0 + c);
                a.s.length[w] = a.s.k;
                a.s.strand[w] = o ? (int8_t)-1 : (int8_t)1;
            }
            base += sum;
            __syncthreads();
        }
    }
}

// First key of every bucket (and n_keys after the last).
__global__ void seed_prefix_kernel(const long long* keys, long long n_keys, int shift, long long n, int32_t* first) {
    for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b <= n; b += (long long)gridDim.x * blockDim.x)
        first[b] = b == n ? (int32_t)n_keys : (int32_t)lower_bound(keys, n_keys, b << shift);
}

int check_index(const gmf_minimizer_index* idx) {
    if (!idx || idx->k < 1 || idx->k > SEED_MAX_K || idx->w < 1 || idx->w > SEED_MAX_W || idx->n_keys < 0)
        return GMF_ERR_INVALID_ARGUMENT;
    if (idx->n_keys > 0 && (!idx->keys || !idx->offsets || !idx->positions)) return GMF_ERR_INVALID_ARGUMENT;
    return GMF_OK;
}

SeedArgs seed_args(const gmf_minimizer_index* idx, int32_t n_reads, const int8_t* codes, const int64_t* read_off,
                   int32_t both) {
    SeedArgs a{};
    a.k = idx->k;
    a.w = idx->w;
    a.n_keys = idx->n_keys;
    a.keys = (const long long*)idx->keys;
    a.offsets = (const long long*)idx->offsets;
    a.positions = idx->positions;
    a.n_reads = n_reads;
    a.codes = codes;
    a.read_off = (const long long*)read_off;
    a.both = both ? 1 : 0;
    return a;
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }
long long tile_slots(int n_reads, long long total) { return total / TILE + n_reads; }

// Workspace: per-read counts, then per tile slot the numbers of selected
// k-mers and anchors, key indices and positions.
size_t carve_tiles(int n_reads, long long total, char* ws, TileArgs& a) {
    const size_t S = (size_t)tile_slots(n_reads, total);
    size_t at = 0;
    auto take = [&](size_t bytes) {
        char* p = ws ? ws + at : nullptr;
        at += up256(bytes);
        return p;
    };
    a.total = total;
    a.slots = (long long)S;
    a.counts = (long long*)take(2 * (size_t)n_reads * 8);
    a.n_anchor = (long long*)take(2 * S * 8);
    a.n_sel = (int32_t*)take(2 * S * 4);
    a.at = (int32_t*)take(2 * S * TILE * 4);
    a.pos = (unsigned short*)take(2 * S * TILE * 2);
    return at;
}

int tile_grid(long long blocks, int per_sm) {
    const long long cap = 148ll * per_sm;
    return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

int seed_grid(int n_reads) {
    const int segs = 2 * n_reads;
    return segs < 148 * 8 ? segs : 148 * 8;
}

}  // namespace

extern "C" int gmf_seed_count(const gmf_minimizer_index* idx, int32_t n_reads, const int8_t* codes,
                              const int64_t* read_off, int32_t both_strands, int64_t* counts, gmf_stream_t stream) {
    GMF_TRY(check_index(idx));
    if (n_reads < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (n_reads == 0) return GMF_OK;
    if (!codes || !read_off || !counts) return GMF_ERR_INVALID_ARGUMENT;
    GMF_BIND_STREAM(stream);
    SeedArgs a = seed_args(idx, n_reads, codes, read_off, both_strands);
    a.counts = (long long*)counts;
    seed_kernel<false><<<seed_grid(n_reads), SEED_THREADS, 0, (cudaStream_t)stream>>>(a);
    return gmf::cuda_status(cudaGetLastError());
}

extern "C" int gmf_seed_fill(const gmf_minimizer_index* idx, int32_t n_reads, const int8_t* codes,
                             const int64_t* read_off, int32_t both_strands, const int64_t* anchor_off,
                             int32_t* read_pos, int32_t* ref_pos, int32_t* length, int8_t* strand,
                             gmf_stream_t stream) {
    GMF_TRY(check_index(idx));
    if (n_reads < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (n_reads == 0) return GMF_OK;
    if (!codes || !read_off || !anchor_off || !read_pos || !ref_pos || !length || !strand)
        return GMF_ERR_INVALID_ARGUMENT;
    GMF_BIND_STREAM(stream);
    SeedArgs a = seed_args(idx, n_reads, codes, read_off, both_strands);
    a.aoff = (const long long*)anchor_off;
    a.read_pos = read_pos;
    a.ref_pos = ref_pos;
    a.length = length;
    a.strand = strand;
    seed_kernel<true><<<seed_grid(n_reads), SEED_THREADS, 0, (cudaStream_t)stream>>>(a);
    return gmf::cuda_status(cudaGetLastError());
}

extern "C" int gmf_seed_prefix_fill(const gmf_minimizer_index* idx, int32_t bits, int32_t* first,
                                    gmf_stream_t stream) {
    GMF_TRY(check_index(idx));
    if (!first || bits < 1 || bits > 2 * idx->k) return GMF_ERR_INVALID_ARGUMENT;
    if (bits > 28 || idx->n_keys > 0x7fffffffll) return GMF_ERR_LIMIT;
    GMF_BIND_STREAM(stream);
    const long long n = 1ll << bits;
    seed_prefix_kernel<<<tile_grid((n + 255) / 256, 16), 256, 0, (cudaStream_t)stream>>>(
        (const long long*)idx->keys, idx->n_keys, 2 * idx->k - bits, n, first);
    return gmf::cuda_status(cudaGetLastError());
}

extern "C" size_t gmf_seed_workspace_bytes(int32_t n_reads, int64_t total_codes) {
    if (n_reads < 0 || total_codes < 0) return 0;
    TileArgs a{};
    return carve_tiles(n_reads, total_codes, nullptr, a);
}

extern "C" int gmf_seed_scan(const gmf_minimizer_index* idx, const gmf_seed_prefix* prefix, int32_t n_reads,
                             const int8_t* codes, const int64_t* read_off, int64_t total_codes, int32_t both_strands,
                             int64_t* anchor_off, int64_t* read_anchor_off, int64_t* totals, void* workspace,
                             size_t workspace_bytes, gmf_stream_t stream_) {
    GMF_TRY(check_index(idx));
    if (n_reads < 0 || total_codes < 0 || !anchor_off || !totals) return GMF_ERR_INVALID_ARGUMENT;
    if (prefix && (!prefix->first || prefix->bits < 1 || prefix->bits > 2 * idx->k)) return GMF_ERR_INVALID_ARGUMENT;
    if (idx->n_keys > 0x7fffffffll) return GMF_ERR_LIMIT;
    if (n_reads > 0 && (!codes || !read_off)) return GMF_ERR_INVALID_ARGUMENT;
    TileArgs a{};
    if (!workspace || workspace_bytes < carve_tiles(n_reads, total_codes, (char*)workspace, a))
        return GMF_ERR_WORKSPACE;
    const cudaStream_t stream = (cudaStream_t)stream_;
    GMF_BIND_STREAM(stream);
    a.s = seed_args(idx, n_reads, codes, read_off, both_strands);
    a.bits = prefix ? prefix->bits : 0;
    a.first = prefix ? prefix->first : nullptr;
    if (n_reads > 0) {
        GMF_CUDA_TRY(cudaMemsetAsync(a.counts, 0, 2 * (size_t)n_reads * 8, stream));
        seed_tile_kernel<<<tile_grid(a.slots, 6), TILE_THREADS, 0, stream>>>(a);
        GMF_CUDA_TRY(cudaGetLastError());
    }
    seed_offsets_kernel<<<1, 1024, 0, stream>>>(n_reads, a.counts, (long long*)anchor_off, (long long*)totals,
                                                (long long*)read_anchor_off);
    return gmf::cuda_status(cudaGetLastError());
}

extern "C" int gmf_seed_emit(const gmf_minimizer_index* idx, int32_t n_reads, const int64_t* read_off,
                             int64_t total_codes, int32_t both_strands, const int64_t* anchor_off, int32_t* read_pos,
                             int32_t* ref_pos, int32_t* length, int8_t* strand, void* workspace,
                             size_t workspace_bytes, gmf_stream_t stream_) {
    GMF_TRY(check_index(idx));
    if (n_reads < 0 || total_codes < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (n_reads == 0) return GMF_OK;
    if (!read_off || !anchor_off || !read_pos || !ref_pos || !length || !strand) return GMF_ERR_INVALID_ARGUMENT;
    TileArgs a{};
    if (!workspace || workspace_bytes < carve_tiles(n_reads, total_codes, (char*)workspace, a))
        return GMF_ERR_WORKSPACE;
    const cudaStream_t stream = (cudaStream_t)stream_;
    GMF_BIND_STREAM(stream);
    a.s = seed_args(idx, n_reads, nullptr, read_off, both_strands);
    a.s.read_pos = read_pos;
    a.s.ref_pos = ref_pos;
    a.s.length = length;
    a.s.strand = strand;
    a.off = (const long long*)anchor_off;
    seed_emit_kernel<<<tile_grid(2 * a.slots, 16), 128, 0, stream>>>(a);
    return gmf::cuda_status(cudaGetLastError());
}
