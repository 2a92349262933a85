// Anchor chaining for sm_100a: strand split + sort, float64 chaining DP,
// chain peeling and primary/secondary selection.
//
// Semantics (GraphMambaFormer):
//   sort      alignment/types.py L144-152   for_strand (+1 then -1) and
//             sorted_by_ref = stable lexsort by (ref_end, read_end)
//   DP        alignment/chaining.py L129-180 chain_dp_numpy: float64
//             ((f[j] + min(min(dq,dr), w_i)) - pen[|dr-dq|]) [+ bonus],
//             argmax = first maximum (lowest j), taken only if > w_i
//   peel      chaining.py L530-576 _backtrack: argsort(-f, stable), claimed
//             mask, partial score f[i] - f[stop]
//   select    chaining.py L579-617 select + _read_overlap
// The log2 penalty comes from a host table, so the device performs only IEEE
// float64 add / subtract / compare in the reference's order and the results
// are bit-identical.
//
// Layout: one CTA per read for sort (a radix sort in shared memory) and
// peel/select, half a warp or a warp per (read, strand) segment for the DP of
// sorted reads: the nearest predecessors first, the rest of the window when
// it could matter.  Segments with weights or bonuses of their own take a warp
// whose lanes own anchors, each finished score broadcast to the window (up to
// 224 predecessors), or, for wider windows, the window sits in a shared-memory
// ring and a warp reduction picks each anchor's predecessor.

#include <float.h>

#include <algorithm>
#include <mutex>

#include "gmf_common.cuh"

namespace gmf {

// ---------------------------------------------------------------------------
// Block-wide bitonic sort of (key, idx) pairs, ascending, ties by idx.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool pair_less(unsigned long long ka, int ia, unsigned long long kb,
                                          int ib) {
    return ka < kb || (ka == kb && ia < ib);
}

__device__ __forceinline__ void bitonic_pair(unsigned long long* key, int* idx, int x, int j, int k) {
    const int y = x | j;  // x has bit j clear
    const bool up = (x & k) == 0;
    const unsigned long long kx = key[x], ky = key[y];
    const int ix = idx[x], iy = idx[y];
    const bool swap = up ? pair_less(ky, iy, kx, ix) : pair_less(kx, ix, ky, iy);
    if (swap) {
        key[x] = ky;
        key[y] = kx;
        idx[x] = iy;
        idx[y] = ix;
    }
}

// Threads take compare-exchange pairs (the p-th index with bit j clear and
// its partner), not elements, so no lane idles.  Stages whose pairs stay
// inside one warp's chunk of the array (j < chunk) need only __syncwarp; only
// the widest strides synchronise the block.  Ends with __syncthreads.
__device__ __forceinline__ void block_bitonic(unsigned long long* key, int* idx, int npow2) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int ch = npow2 / nw;
    if (ch < 64) ch = 64;
    if (ch > npow2) ch = npow2;
    const int n_chunks = npow2 / ch;
    bool block_synced = true;
    for (int k = 2; k <= npow2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= ch) {
                if (!block_synced) __syncthreads();
                for (int p = threadIdx.x; p < (npow2 >> 1); p += blockDim.x)
                    bitonic_pair(key, idx, ((p & ~(j - 1)) << 1) | (p & (j - 1)), j, k);
                __syncthreads();
                block_synced = true;
            } else {
                for (int c = wid; c < n_chunks; c += nw) {
                    const int base = c * ch;
                    for (int p = lane; p < (ch >> 1); p += 32)
                        bitonic_pair(key, idx, base + (((p & ~(j - 1)) << 1) | (p & (j - 1))), j, k);
                }
                __syncwarp();
                block_synced = false;
            }
        }
    }
    __syncthreads();
}

__host__ __device__ inline int next_pow2(int n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Order-preserving map of a double onto uint64 (ascending), -0.0 == +0.0.
__device__ __forceinline__ unsigned long long ordered_bits(double v) {
    if (v == 0.0) v = 0.0;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// ---------------------------------------------------------------------------
// Sort: per read, strand +1 anchors then strand -1 anchors, each by
// (ref_end, read_end, original index).
// ---------------------------------------------------------------------------
struct SortArgs {
    int32_t n_reads;
    const int64_t* read_off;
    const int32_t* read_pos;
    const int32_t* ref_pos;
    const int32_t* length;
    const int8_t* strand;
    int32_t* perm;
    int32_t* n_plus;
    int32_t* n_minus;
    int32_t* read_end_s;
    int32_t* ref_end_s;
    int32_t* len_s;            // sorted lengths (workspace), or null
    int64_t cap;               // anchors the sorted outputs can hold (-1: caller-sized)
    int64_t key_cap;           // anchors the caller's workspace covers (reads beyond SORT_CAP need it)
    int* err;
    const double* lut;         // with min_pen: the penalty table, for the DP's bound
    int max_gap;
    double* min_pen;           // its smallest entry, or null
};

// Radix sort of a read's anchors in shared memory: 16-bit indices by 8-bit
// digits of a 32-bit key, least significant first.  Every pass is stable, so
// equal keys keep the input order, which is the reference's last tie-breaker.
// The key is the strand and ref_end (less the read's smallest); read_end needs
// passes of its own only when the anchors do not come in (strand, read_end)
// order, which is how seeding writes them.  A pass ranks each warp's run of
// anchors row by row of 32 (lanes of equal digit found by a match), turns the
// warps' digit counts into offsets, and scatters the indices.
//
// What bounds it is the latency of a pass's rows; a bitonic sort of (key,
// index) pairs took 78 stages for 4,096 keys (199,000 warp instructions for a
// 15 kb read's 2,700 anchors) and went through global memory beyond that.
// Measured on one B200: one 15 kb read 89 -> 32 us (4 of them the table's
// minimum), 5,000 of them 1,275 -> 341 us, 1,000 reads of 10,000 anchors 2,172
// -> 299 us.  The digit passes want 5 blocks an SM (48 registers; with 4, 5,000
// reads take 10% longer).
constexpr int SORT_CAP = 4096;      // anchors a 256-thread block sorts; larger reads take 1,024 threads
constexpr int SORT_CAP_BIG = 16384;
constexpr int SORT_ROWS = 16;       // rows of 32 a warp takes at most (both: 512 anchors a warp)
static_assert(SORT_CAP_BIG >= GMF_MAX_READ_ANCHORS, "a read's anchors fit the large block");
// Up to RANK_CAP anchors are placed by counting the smaller ones, a thread
// each, which takes less than the digit passes (2,000 reads in a whole call, by
// digits / by counting: of 90 anchors 125 / 96 us, of 200 133 / 126, of 250 145
// / 148).
constexpr int RANK_CAP = 224;

template <int T>
struct SortSmem {
    unsigned short hist[T / 32][256];
    unsigned bin[256];
    unsigned red[T / 32];
    unsigned red2[T / 32];
};

template <int T, int CAP>
constexpr size_t sort_smem_size() {
    return (size_t)CAP * 8 + sizeof(SortSmem<T>);
}

// One stable pass by bits [shift, shift + 8) of key[]: src -> dst.
template <int T>
__device__ __forceinline__ void radix_pass(SortSmem<T>& S, const unsigned* key, const unsigned short* src,
                                           unsigned short* dst, int n, int shift) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int rows = (n + T - 1) / T;  // per warp
    const int first = w * rows * 32;
    unsigned short* h = S.hist[w];
#pragma unroll
    for (int x = 0; x < 4; ++x) reinterpret_cast<unsigned*>(h)[lane + 32 * x] = 0u;
    __syncwarp();
    unsigned at[SORT_ROWS];  // digit and place among the warp's anchors of that digit
#pragma unroll
    for (int i = 0; i < SORT_ROWS; ++i) {
        at[i] = 0u;
        if (i < rows) {
            const int x = first + 32 * i + lane;
            const unsigned d = x < n ? (key[src[x]] >> shift) & 255u : 256u;
            const unsigned same = __match_any_sync(FULL_MASK, d);
            const unsigned rank = __popc(same & lt);
            unsigned base = 0;
            if (x < n) base = h[d];
            __syncwarp();
            if (x < n && rank == 0) h[d] = (unsigned short)(base + __popc(same));
            __syncwarp();
            at[i] = d << 16 | (base + rank);
        }
    }
    __syncthreads();
    // offsets: digit by digit, within a digit warp by warp
    if (tid < 256) {
        unsigned run = 0;
#pragma unroll 8
        for (int v = 0; v < T / 32; ++v) {
            const unsigned c = S.hist[v][tid];
            S.hist[v][tid] = (unsigned short)run;
            run += c;
        }
        unsigned incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) S.red[w] = incl;
        S.bin[tid] = incl - run;
    }
    __syncthreads();
    if (tid < 256) {
        unsigned before = 0;
        for (int v = 0; v < w; ++v) before += S.red[v];
        S.bin[tid] += before;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SORT_ROWS; ++i) {
        const int x = first + 32 * i + lane;
        if (i < rows && x < n) {
            const unsigned d = at[i] >> 16;
            dst[S.bin[d] + h[d] + (at[i] & 0xFFFFu)] = src[x];
        }
    }
    __syncthreads();
}

template <int T>
__device__ __forceinline__ unsigned block_max(SortSmem<T>& S, unsigned v, unsigned* red) {
    v = __reduce_max_sync(FULL_MASK, v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (int w = 1; w < T / 32; ++w) v = max(v, red[w]);
    return v;
}

__device__ __forceinline__ unsigned bits_of(unsigned v) { return 32u - __clz(v); }

__device__ __forceinline__ void sort_small_read(const SortArgs& a, int r, int n) {
    extern __shared__ __align__(16) unsigned sort_smem[];
    unsigned long long* key = reinterpret_cast<unsigned long long*>(sort_smem);
    const int x = threadIdx.x;
    const int64_t a0 = a.read_off[r];
    unsigned long long mine = ~0ull;  // (strand group, ref_end, read_end)
    int len = 0;
    if (x < n) {
        const int8_t s = a.strand[a0 + x];
        len = a.length[a0 + x];
        mine = (s == 1 ? 0ull : (s == -1 ? 1ull : 2ull)) << 62 |
               (unsigned long long)((unsigned)(a.ref_pos[a0 + x] + len) & 0x7fffffffu) << 31 |
               ((unsigned)(a.read_pos[a0 + x] + len) & 0x7fffffffu);
        key[x] = mine;
    }
    const int n0 = __syncthreads_count(x < n && mine >> 62 == 0);
    const int m = __syncthreads_count(x < n && mine >> 62 < 2);
    if (x < n && mine >> 62 < 2) {
        int rank = 0;
#pragma unroll 8
        for (int y = 0; y < n; ++y) rank += key[y] < mine || (key[y] == mine && y < x);
        a.perm[a0 + rank] = x;
        if (a.len_s) a.len_s[a0 + rank] = len;
        a.ref_end_s[a0 + rank] = (int32_t)((mine >> 31) & 0x7fffffffu);
        a.read_end_s[a0 + rank] = (int32_t)(mine & 0x7fffffffu);
    }
    if (x == 0) {
        a.n_plus[r] = n0;
        a.n_minus[r] = m - n0;
    }
}

// The penalty table's smallest entry, by a block of 256 threads.
__device__ __forceinline__ void smallest_penalty(const double* __restrict__ lut, int max_gap, double* out) {
    __shared__ double s_min[8];
    double m = INFINITY;
#pragma unroll 8
    for (int x = threadIdx.x; x <= max_gap; x += 256) m = fmin(m, __ldg(&lut[x]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(FULL_MASK, m, o));
    if ((threadIdx.x & 31) == 0) s_min[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int x = 1; x < 8; ++x) m = fmin(m, s_min[x]);
        *out = m;
    }
}

template <int T>
__device__ void sort_read(const SortArgs& a, int r, int n, unsigned* key, unsigned short* ia, unsigned short* ib,
                          SortSmem<T>& S, int* cnt) {
    const int tid = threadIdx.x;
    const int64_t a0 = a.read_off[r];
    const int32_t* rp = a.read_pos + a0;
    const int32_t* fp = a.ref_pos + a0;
    const int32_t* ln = a.length + a0;
    const int8_t* sd = a.strand + a0;
    auto group = [&](int x) { return sd[x] == 1 ? 0u : (sd[x] == -1 ? 1u : 2u); };
    auto read_end = [&](int x) { return (unsigned)(rp[x] + ln[x]) & 0x7fffffffu; };
    if (T == 256 && n <= RANK_CAP) {
        sort_small_read(a, r, n);
        return;
    }
    if (tid < 3) cnt[tid] = 0;
    __syncthreads();
    // extremes, strand counts, and whether the anchors come in (strand, read_end) order
    unsigned hi = 0, lo_c = 0, re_max = 0, c0 = 0, c1 = 0;  // lo_c: complement of the smallest
    bool unordered = false;
    for (int x = tid; x < n; x += T) {
        const unsigned fe = (unsigned)(fp[x] + ln[x]) & 0x7fffffffu, re = read_end(x), g = group(x);
        key[x] = fe;
        ia[x] = (unsigned short)x;
        hi = max(hi, fe);
        lo_c = max(lo_c, ~fe);
        re_max = max(re_max, re);
        c0 += g == 0u;
        c1 += g == 1u;
        if (x > 0) {
            const unsigned gp = group(x - 1);
            unordered |= gp > g || (gp == g && read_end(x - 1) > re);
        }
    }
    c0 = __reduce_add_sync(FULL_MASK, c0);
    c1 = __reduce_add_sync(FULL_MASK, c1);
    if ((tid & 31) == 0) {
        if (c0) atomicAdd(&cnt[0], (int)c0);
        if (c1) atomicAdd(&cnt[1], (int)c1);
    }
    hi = block_max<T>(S, hi, S.red);
    const unsigned lo = ~block_max<T>(S, lo_c, S.red2);
    unordered = __syncthreads_or(unordered);
    const int n0 = cnt[0], m = cnt[0] + cnt[1];
    const bool mixed = n0 != n && cnt[1] != n;  // several strands
    unsigned short *src = ia, *dst = ib;
    auto passes = [&](int bits) {
        for (int b = 0; b < bits; b += 8) {
            radix_pass<T>(S, key, src, dst, n, b);
            unsigned short* t = src;
            src = dst;
            dst = t;
        }
    };
    if (unordered) {
        re_max = block_max<T>(S, re_max, S.red);
        __syncthreads();
        for (int x = tid; x < n; x += T) key[x] = read_end(x);
        __syncthreads();
        passes((int)bits_of(re_max));
    }
    const int nb = (int)bits_of(hi - lo);
    const bool fold = mixed && nb <= 30;
    __syncthreads();
    for (int x = tid; x < n; x += T)
        key[x] = (((unsigned)(fp[x] + ln[x]) & 0x7fffffffu) - lo) | (fold ? group(x) << nb : 0u);
    __syncthreads();
    passes(nb + (fold ? 2 : 0));
    if (mixed && !fold) {
        for (int x = tid; x < n; x += T) key[x] = group(x);
        __syncthreads();
        passes(2);
    }
    for (int x = tid; x < m; x += T) {
        const int id = src[x];
        a.perm[a0 + x] = id;
        if (a.len_s) a.len_s[a0 + x] = ln[id];
        a.ref_end_s[a0 + x] = (int32_t)((unsigned)(fp[id] + ln[id]) & 0x7fffffffu);
        a.read_end_s[a0 + x] = (int32_t)read_end(id);
    }
    if (tid == 0) {
        a.n_plus[r] = n0;
        a.n_minus[r] = m - n0;
    }
}

// Anchors of read r, or -1 (with the error noted) when the read cannot be
// sorted: too many anchors for one read, or beyond what the workspace holds.
// Such a read gets no sorted anchors (so no chains).  (gmf_chain_sort refuses
// reads of more than SORT_CAP anchors that its workspace does not cover, which
// once held their keys: a caller may count on the error.)
__device__ __forceinline__ int sort_count(const SortArgs& a, int r, int* error) {
    const int64_t a0 = a.read_off[r];
    const int n = (int)(a.read_off[r + 1] - a0);
    *error = 0;
    if (n > GMF_MAX_READ_ANCHORS) *error = 1;
    else if (a.cap >= 0 && a.read_off[r + 1] > a.cap) *error = 4;
    else if (n > SORT_CAP && 2 * a0 + next_pow2(n) > 2 * a.key_cap) *error = 2;
    return *error ? -1 : n;
}

__global__ void __launch_bounds__(256, 5) chain_sort_kernel(SortArgs a) {
    extern __shared__ __align__(16) unsigned sort_smem[];
    __shared__ int cnt[3];
    const int r = blockIdx.x;
    if (r == 0 && a.min_pen) smallest_penalty(a.lut, a.max_gap, a.min_pen);  // not by every block of the DP
    int error;
    const int n = sort_count(a, r, &error);
    if (n < 0) {
        if (threadIdx.x == 0) {
            a.n_plus[r] = 0;
            a.n_minus[r] = 0;
            if (a.err) atomicOr(a.err, error);
        }
        return;
    }
    if (n > SORT_CAP) return;  // chain_sort_big_kernel
    unsigned short* ia = reinterpret_cast<unsigned short*>(sort_smem + SORT_CAP);
    sort_read<256>(a, r, n, sort_smem, ia, ia + SORT_CAP,
                   *reinterpret_cast<SortSmem<256>*>(ia + 2 * SORT_CAP), cnt);
}

// Reads of more than SORT_CAP anchors: a block looks through every gridDim-th
// read and sorts the large ones.
__global__ void __launch_bounds__(1024) chain_sort_big_kernel(SortArgs a) {
    extern __shared__ __align__(16) unsigned sort_smem[];
    __shared__ int cnt[3];
    __shared__ int n_found, found[1024];
    unsigned short* ia = reinterpret_cast<unsigned short*>(sort_smem + SORT_CAP_BIG);
    SortSmem<1024>& S = *reinterpret_cast<SortSmem<1024>*>(ia + 2 * SORT_CAP_BIG);
    for (int64_t first = blockIdx.x; first < a.n_reads; first += (int64_t)gridDim.x * 1024) {
        if (threadIdx.x == 0) n_found = 0;
        __syncthreads();
        const int64_t r = first + (int64_t)threadIdx.x * gridDim.x;
        int error;
        if (r < a.n_reads && sort_count(a, (int)r, &error) > SORT_CAP) found[atomicAdd(&n_found, 1)] = (int)r;
        __syncthreads();
        for (int k = 0; k < n_found; ++k) {
            const int q = found[k];
            sort_read<1024>(a, q, (int)(a.read_off[q + 1] - a.read_off[q]), sort_smem, ia, ia + SORT_CAP_BIG, S, cnt);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Chaining DP: one warp per segment of sorted anchors.
// ---------------------------------------------------------------------------
struct DpArgs {
    // segment source: either explicit rows (row_off) or sorted reads
    int32_t n_segments;
    const int64_t* row_off;   // rows mode
    const int64_t* read_off;  // reads mode
    const int32_t* n_plus;
    const int32_t* n_minus;
    const int32_t* read_end;
    const int32_t* ref_end;
    const double* weight;    // NULL: anchor length (reads mode), via length_s
    const int32_t* length;   // original lengths (reads mode, weight == NULL)
    const int32_t* len_s;    // sorted lengths, or null: length[perm[]]
    const int32_t* perm;     // reads mode
    const double* bonus;
    int32_t lookback;
    int32_t max_gap;
    const double* lut;
    int32_t lut_len;
    double* f;
    int32_t* parent;
    int32_t ring;            // ring entries per warp (power of two > lookback)
    const double* min_pen;   // near: the table's smallest penalty
    bool near;               // sorted by this call with lengths as weights: at most GMF_MAX_READ_ANCHORS a segment
    int64_t cap;             // reads mode: anchors f / parent hold (-1: caller-sized)
};

__device__ __forceinline__ void seg_range(const DpArgs& a, int s, int64_t& start, int& n) {
    if (a.row_off) {
        start = a.row_off[s];
        n = (int)(a.row_off[s + 1] - start);
    } else {
        const int r = s >> 1;
        const int64_t a0 = a.read_off[r];
        if ((s & 1) == 0) {
            start = a0;
            n = a.n_plus[r];
        } else {
            start = a0 + a.n_plus[r];
            n = a.n_minus[r];
        }
        if (a.cap >= 0 && start + n > a.cap) n = 0;  // beyond the workspace: skipped
    }
}

__global__ void __launch_bounds__(128) chain_dp_kernel(DpArgs a) {
    extern __shared__ double dp_smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    const int R = a.ring;
    const int mask = R - 1;
    double* rf = dp_smem + (size_t)wib * R * 2;  // f ring, then (read_end, ref_end) as int2
    int2* rc = reinterpret_cast<int2*>(rf + R);
    const int lb = a.lookback > 1 ? a.lookback : 1;
    for (int s = blockIdx.x * wpb + wib; s < a.n_segments; s += gridDim.x * wpb) {
        int64_t st;
        int n;
        seg_range(a, s, st, n);
        int64_t r0 = 0;
        if (!a.row_off) r0 = a.read_off[s >> 1];
        for (int i = 0; i < n; ++i) {
            const int64_t gi = st + i;
            const int qi = a.read_end[gi];
            const int ri = a.ref_end[gi];
            double wi;
            if (a.weight)
                wi = a.weight[gi];
            else
                wi = (double)a.length[r0 + a.perm[gi]];
            const int lo = i - lb > 0 ? i - lb : 0;
            double best = -DBL_MAX;
            int bj = -1;
            bool any = false;
            for (int j = lo + lane; j < i; j += 32) {
                const int2 c = rc[j & mask];
                const int dq = qi - c.x;
                const int dr = ri - c.y;
                double sc;
                if (dq > 0 && dr > 0 && dq <= a.max_gap && dr <= a.max_gap) {
                    any = true;
                    const double mn = (double)(dq < dr ? dq : dr);
                    const double adv = mn < wi ? mn : wi;
                    const int gap = dr > dq ? dr - dq : dq - dr;
                    sc = __dsub_rn(__dadd_rn(rf[j & mask], adv), __ldg(&a.lut[gap]));
                    if (a.bonus) sc = __dadd_rn(sc, __ldg(&a.bonus[gi * lb + (lb - (i - lo)) + (j - lo)]));
                } else {
                    sc = -1e30;
                }
                if (bj < 0 || sc > best) {
                    best = sc;
                    bj = j;
                }
            }
            any = __any_sync(FULL_MASK, any);
            double fi = wi;
            int pi = -1;
            if (any) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const double ob = __shfl_xor_sync(FULL_MASK, best, o);
                    const int oj = __shfl_xor_sync(FULL_MASK, bj, o);
                    const bool take = (oj >= 0) && (bj < 0 || ob > best || (ob == best && oj < bj));
                    if (take) {
                        best = ob;
                        bj = oj;
                    }
                }
                if (best > wi) {
                    fi = best;
                    pi = bj;
                }
            }
            if (lane == 0) {
                rf[i & mask] = fi;
                rc[i & mask] = make_int2(qi, ri);
                a.f[gi] = fi;
                a.parent[gi] = pi;
            }
            __syncwarp();
        }
    }
}

// The same recurrence with the anchors owned by lanes: lane l holds anchor
// 32(b+k) + l of K consecutive blocks of 32 (K - 1 blocks cover the window).
// Step t finalises anchor t (its owner's running maximum against w_t),
// broadcasts (f_t, read_end_t, ref_end_t), and every anchor i with
// 1 <= i - t <= lb folds the candidate of predecessor t into its running
// maximum.  Candidates arrive in ascending j and replace the maximum only when
// strictly larger, so the first maximum (lowest j) wins as in the reference;
// each candidate is the same float64 add / subtract.  After 32 steps the
// finished block is stored (coalesced) and the next block is loaded.
template <bool WEIGHT>
__device__ __forceinline__ void dp_load_slot(const DpArgs& a, int64_t st, int64_t r0, int i, int n,
                                             int& q, int& r, double& w, int& wl) {
    if (i < n) {
        const int64_t gi = st + i;
        q = a.read_end[gi];
        r = a.ref_end[gi];
        if (WEIGHT) {
            w = a.weight[gi];
        } else {
            wl = a.len_s ? a.len_s[gi] : a.length[r0 + a.perm[gi]];
            w = (double)wl;
        }
    } else {
        q = 0;
        r = 0;
        w = 0.0;
        wl = 0;
    }
}

// Every candidate of a step is computed without branches (the table index is
// clamped so that out-of-window pairs read in bounds) and folded in under one
// predicate.  The running maxima start at -inf: the first valid candidate
// (finite) always replaces it, as the reference's first maximum.
template <int K, bool WEIGHT, bool BONUS>
__global__ void __launch_bounds__(128) chain_dp_bcast_kernel(DpArgs a) {
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    const int lb = a.lookback > 1 ? a.lookback : 1;
    const unsigned mg = a.max_gap > 0 ? (unsigned)a.max_gap : 0u;
    const double* __restrict__ lut = a.lut;
    // reads mode: warps take every read's longer strand first, then the
    // shorter ones, so a block's warps have similar work and the short
    // segments fill the tail
    const int n_reads = a.n_segments >> 1;
    for (int g = blockIdx.x * wpb + wib; g < a.n_segments; g += gridDim.x * wpb) {
        int s = g;
        if (!a.row_off) {
            const int r = g < n_reads ? g : g - n_reads;
            const int minus_longer = a.n_minus[r] > a.n_plus[r] ? 1 : 0;
            s = 2 * r + (g < n_reads ? minus_longer : 1 - minus_longer);
        }
        int64_t st;
        int n;
        seg_range(a, s, st, n);
        if (n <= 0) continue;
        const int64_t r0 = a.row_off ? 0 : a.read_off[s >> 1];
        int q[K], rr[K], bj[K], wl[K];
        double w[K], best[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            dp_load_slot<WEIGHT>(a, st, r0, 32 * k + lane, n, q[k], rr[k], w[k], wl[k]);
            best[k] = -INFINITY;
            bj[k] = -1;
        }
        for (int base = 0; base < n; base += 32) {
            const int steps = n - base < 32 ? n - base : 32;
            bool live[K];
#pragma unroll
            for (int k = 0; k < K; ++k) live[k] = base + 32 * k + lane < n;
            for (int u = 0; u < steps; ++u) {
                const double fo = best[0] > w[0] ? best[0] : w[0];
                const double ft = __shfl_sync(FULL_MASK, fo, u);
                const int qt = __shfl_sync(FULL_MASK, q[0], u);
                const int rt = __shfl_sync(FULL_MASK, rr[0], u);
                const int t = base + u;
                const int lu = lane - u;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    // a block none of whose anchors reaches back to t is skipped
                    if (32 * k - u > lb) continue;
                    const int d = 32 * k + lu;
                    const int dq = q[k] - qt;
                    const int dr = rr[k] - rt;
                    const bool ok = live[k] && (unsigned)(d - 1) < (unsigned)lb &&
                                    (unsigned)(dq - 1) < mg && (unsigned)(dr - 1) < mg;
                    const int mn = dq < dr ? dq : dr;
                    double adv;
                    if (WEIGHT) {
                        const double mnd = (double)mn;
                        adv = mnd < w[k] ? mnd : w[k];
                    } else {
                        adv = (double)(mn < wl[k] ? mn : wl[k]);
                    }
                    unsigned gap = (unsigned)(dr > dq ? dr - dq : dq - dr);
                    gap = gap < mg ? gap : mg;
                    double sc = __dsub_rn(__dadd_rn(ft, adv), __ldg(&lut[gap]));
                    if (BONUS) {
                        const int64_t bi = ok ? (st + base + 32 * k + lane) * lb + (lb - d) : 0;
                        sc = __dadd_rn(sc, __ldg(&a.bonus[bi]));
                    }
                    if (ok && sc > best[k]) {
                        best[k] = sc;
                        bj[k] = t;
                    }
                }
            }
            if (live[0]) {
                const bool take = best[0] > w[0];
                a.f[st + base + lane] = take ? best[0] : w[0];
                a.parent[st + base + lane] = take ? bj[0] : -1;
            }
#pragma unroll
            for (int k = 0; k + 1 < K; ++k) {
                q[k] = q[k + 1];
                rr[k] = rr[k + 1];
                w[k] = w[k + 1];
                wl[k] = wl[k + 1];
                best[k] = best[k + 1];
                bj[k] = bj[k + 1];
            }
            dp_load_slot<WEIGHT>(a, st, r0, base + 32 * K + lane, n, q[K - 1], rr[K - 1], w[K - 1], wl[K - 1]);
            best[K - 1] = -INFINITY;
            bj[K - 1] = -1;
        }
    }
}

// The same recurrence with the nearest predecessors first, for sorted reads
// whose weights are their lengths (no bonus).  A group of G lanes runs one
// segment, G anchors (a block) at a time: every lane first computes, for its
// own anchor, advance and penalty against the NEAR nearest predecessors --
// nothing of that depends on f -- and then all lanes of the group step
// through the block's anchors together, each anchor scoring its NEAR nearest
// predecessors from shared memory, oldest first, so that the first maximum
// wins and only two additions and a compare lie between f[i-1] and f[i].
//
// Predecessors beyond the nearest are scored only when they could matter:
// none of them scores more than (the largest f among them) + w_i - (the
// smallest penalty), float64 rounding being monotone, and on a chain f grows
// by several units per anchor, so that bound (with the largest f of all older
// anchors) nearly always lies below the best near candidate.  Otherwise the
// group's lanes score the rest of the window, oldest first; an older
// candidate wins a tie.
//
// What bounds it is that chain, one segment being one serial scan: the
// broadcast form above scores the whole window (98 instructions and ~480
// cycles an anchor for a window of 50, 8 blocks of 32 for 200).  A pull form
// with one candidate per lane and two warp reductions per anchor took 100
// instructions and 380 cycles.  Measured on one B200, DP kernel alone: one
// 15 kb HiFi read 675 -> 263 us, 5,000 of them 1,874 -> 825 us (window 50),
// 1,000 reads of 50-100 kb 5,011 -> 1,029 us (window 200).
//
// Anchors of repeats, on several diagonals at once, have their predecessors
// beyond the nearest, and the rest of the window one anchor at a time takes
// ~1,500 cycles.  So where the bound fails often, the next block scores whole
// windows instead (dp_whole_block): every lane folds its own anchor's
// candidates of the blocks before in one pass, which no f of this block holds
// up, and the block's own as each of its f is broadcast.  It costs ~200 cycles
// an anchor (window 64), a little more than the nearest alone, and so takes
// over at 12 failures in 32 anchors: with 4 a read of one chain with gaps was
// up to 9% slower, with 12 none by more than 2%.  The first block, whose whole
// window is the block itself, is done so as well.  Whole calls (sort, DP and
// peel) on one B200, the broadcast form / the nearest alone / both: one read of
// 2,500 anchors on five diagonals 585 / 966 / 466 us, random anchors 999 / 2,119
// / 823, 9,157 / 16,075 / 5,249 with a window of 1,000; 2,000 reads of 1,500
// anchors on five diagonals 999 / 1,286 / 830.
__device__ __forceinline__ double int_to_double(int x) {  // exact: one add instead of a conversion
    return __hiloint2double(0x43300000, x ^ (int)0x80000000) - 4503601774854144.0;  // 2^52 + 2^31
}

// Advance and penalty of a predecessor (dq, dr behind the anchor), infinite
// penalty when the pair is out of range.
__device__ __forceinline__ double2 dp_pair(int dq, int dr, int wl, bool in, unsigned mg,
                                           const double* __restrict__ lut) {
    const bool ok = in && (unsigned)(dq - 1) < mg && (unsigned)(dr - 1) < mg;
    const int mn = dq < dr ? dq : dr;
    const unsigned gap = (unsigned)(dr > dq ? dr - dq : dq - dr);
    const double pen = __ldg(&lut[gap < mg ? gap : mg]);
    return make_double2(ok ? int_to_double(mn < wl ? mn : wl) : 0.0, ok ? pen : INFINITY);
}

constexpr int NEAR = 4;
constexpr double NEAR_SLACK = 0.015625;  // of the bound, for a candidate's two roundings: |f| < 2^14 anchors * 2^31
constexpr int WHOLE_FROM = 12;       // of 32 anchors, see above
constexpr int NEAR_MAX_GAP = 16384;  // one block of the sort reads the whole penalty table for its minimum
constexpr int NEAR_WARPS = 2;        // per block: small blocks spread the long segments over the SMs

// What the next block needs to know of the anchors before it.
struct Tail {
    double f1, f2, f3, f4;  // f of the four before, nearest first
    double older;           // largest f before those
    int far;                // anchors of the last block to which an older predecessor may have mattered
};

// A block of G anchors per group with their whole windows (q, r, wl: the
// lane's anchor; qr_at, f_at: bytes of the group's rings in shared memory).
// Not inlined, so that it takes no registers from the nearest-first loop.
template <int G>
__device__ __noinline__ Tail dp_whole_block(int qr_at, int f_at, int rm, int base, int n, int lb, unsigned mg,
                                            const double* __restrict__ lut, int q, int r, int wl, double min_pen,
                                            double* f_out, int32_t* parent_out, Tail t) {
    extern __shared__ double2 near_smem[];
    const int2* s_qr = reinterpret_cast<const int2*>(reinterpret_cast<unsigned char*>(near_smem) + qr_at);
    double* s_f = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(near_smem) + f_at);
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), mine = base + gl;
    const double w = int_to_double(wl);
    double bs = -INFINITY;
    int bj = -1;
    auto fold = [&](int j, const int2& c, double fj, bool in) {
        const int dq = q - c.x, dr = r - c.y;
        const int mn = dq < dr ? dq : dr;
        const unsigned gap = (unsigned)(dr > dq ? dr - dq : dq - dr);
        const double sc = __dsub_rn(__dadd_rn(fj, int_to_double(mn < wl ? mn : wl)), __ldg(&lut[gap < mg ? gap : mg]));
        if (in && (unsigned)(dq - 1) < mg && (unsigned)(dr - 1) < mg && sc > bs) {
            bs = sc;
            bj = j;
        }
    };
#pragma unroll 8
    for (int j = base > lb ? base - lb : 0; j < base; ++j) fold(j, s_qr[j & rm], s_f[j & rm], j >= mine - lb);
#pragma unroll 4
    for (int u = 0; u < G; ++u) {
        const double fu = __shfl_sync(FULL_MASK, bs > w ? bs : w, u, G);
        fold(base + u, s_qr[(base + u) & rm], fu, gl > u && gl - u <= lb);
    }
    const double fi = bs > w ? bs : w;
    s_f[mine & rm] = fi;
    if (mine < n) {
        f_out[mine] = fi;
        parent_out[mine] = bs > w ? bj : -1;
    }
    // how often the nearest alone would not have done: the largest f before each anchor's nearest four, in the bound
    double up_to = mine < n ? fi : -INFINITY;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const double v = __shfl_up_sync(FULL_MASK, up_to, o, G);
        if (gl >= o && v > up_to) up_to = v;
    }
    double before = t.older;
    if (base > 0) {
        before = gl >= 1 ? fmax(before, t.f4) : before;
        before = gl >= 2 ? fmax(before, t.f3) : before;
        before = gl >= 3 ? fmax(before, t.f2) : before;
        before = gl >= 4 ? fmax(before, t.f1) : before;
    }
    const double in_block = __shfl_up_sync(FULL_MASK, up_to, NEAR + 1, G);
    if (gl > NEAR) before = fmax(before, in_block);
    const unsigned m = __ballot_sync(FULL_MASK, mine < n && before + (w - min_pen + NEAR_SLACK) >= fi);
    t.far = __popc(G == 32 ? m : (m >> (lane & ~(G - 1))) & ((1u << (G & 31)) - 1u));
    t.older = __shfl_sync(FULL_MASK, fmax(before, up_to), G - 1 - NEAR, G);
    t.f1 = __shfl_sync(FULL_MASK, fi, G - 1, G);
    t.f2 = __shfl_sync(FULL_MASK, fi, G - 2, G);
    t.f3 = __shfl_sync(FULL_MASK, fi, G - 3, G);
    t.f4 = __shfl_sync(FULL_MASK, fi, G - 4, G);
    return t;
}

__host__ __device__ inline size_t near_smem_bytes(int G, int ring) {  // per group
    return (size_t)G * (NEAR * 16 + 16 + 8) + (size_t)ring * 16;
}

template <int G>
__global__ void __launch_bounds__(32 * NEAR_WARPS) chain_dp_near_kernel(DpArgs a) {
    extern __shared__ double2 near_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, gl = lane & (G - 1);
    constexpr int GPW = 32 / G, UNROLL = 8;
    const int R = a.ring, rm = R - 1;  // R is a multiple of G: a block's entries never wrap
    unsigned char* sm = reinterpret_cast<unsigned char*>(near_smem) +
                        (size_t)(threadIdx.x / G) * near_smem_bytes(G, R);
    double2* s_pair = reinterpret_cast<double2*>(sm);              // [G][NEAR] (advance, penalty), nearest first
    double2* s_w = s_pair + G * NEAR;                              // [G] (weight, weight - smallest penalty + slack)
    double* s_f = reinterpret_cast<double*>(s_w + G);              // ring of f
    int2* s_qr = reinterpret_cast<int2*>(s_f + R);                 // ring of (read_end, ref_end)
    const int ring_at = (int)(reinterpret_cast<unsigned char*>(s_f) - reinterpret_cast<unsigned char*>(near_smem));
    const int qr_at = (int)(reinterpret_cast<unsigned char*>(s_qr) - reinterpret_cast<unsigned char*>(near_smem));
    int* s_p = reinterpret_cast<int*>(s_qr + R);                   // [G] age of a predecessor beyond the nearest, else 0;
                                                                   // [G] the number of anchors that looked for one
    const int lb = a.lookback > 1 ? a.lookback : 1;
    const unsigned mg = a.max_gap > 0 ? (unsigned)a.max_gap : 0u;
    const double* __restrict__ lut = a.lut;
    const double min_pen = *a.min_pen;  // smallest penalty a candidate can take

    const int n_reads = a.n_segments >> 1;
    const int n_groups = gridDim.x * NEAR_WARPS * GPW;
    for (int g0 = (blockIdx.x * NEAR_WARPS + wib) * GPW; g0 < a.n_segments; g0 += n_groups) {
        const int g = g0 + lane / G;
        int64_t st = 0, r0 = 0;
        int n = 0;
        if (g < a.n_segments) {
            // every read's longer strand first, then the shorter ones
            const int r = g < n_reads ? g : g - n_reads;
            const int minus_longer = a.n_minus[r] > a.n_plus[r] ? 1 : 0;
            seg_range(a, 2 * r + (g < n_reads ? minus_longer : 1 - minus_longer), st, n);
            r0 = a.read_off[r];
        }
        const int blocks = __reduce_max_sync(FULL_MASK, (n + G - 1) / G);
        double f1 = 0.0, f2 = 0.0, f3 = 0.0, f4 = 0.0;  // f of the four anchors before
        double older = -INFINITY;                       // largest f before those
        bool whole = true;                              // the block's anchors score their whole window
        int q, r, wl;
        double unused;
        dp_load_slot<false>(a, st, r0, gl, n, q, r, unused, wl);
        for (int b = 0; b < blocks; ++b) {
            const int base = b * G, mine = base + gl;
            double* f_at = s_f + (base & rm);
            __syncwarp();
            s_qr[mine & rm] = make_int2(q, r);
            s_p[gl] = 0;
            if (gl == 0) s_p[G] = 0;
            __syncwarp();
            if (whole) {  // uniform over the warp
                Tail t{f1, f2, f3, f4, older, 0};
                const int bq = q, br = r, bl = wl;
                dp_load_slot<false>(a, st, r0, mine + G, n, q, r, unused, wl);  // the next block
                t = dp_whole_block<G>(qr_at, ring_at, rm, base, n, lb, mg, lut, bq, br, bl, min_pen, a.f + st,
                                      a.parent + st, t);
                f1 = t.f1;
                f2 = t.f2;
                f3 = t.f3;
                f4 = t.f4;
                older = t.older;
                whole = __any_sync(FULL_MASK, t.far >= WHOLE_FROM * G / 32);
                continue;
            }
#pragma unroll
            for (int d = 1; d <= NEAR; ++d) {
                const int2 c = s_qr[(mine - d) & rm];
                s_pair[gl * NEAR + d - 1] = dp_pair(q - c.x, r - c.y, wl, d <= mine && d <= lb && mine < n, mg, lut);
            }
            {
                const double w = int_to_double(wl);
                s_w[gl] = make_double2(w, mine < n ? w - min_pen + NEAR_SLACK : -INFINITY);
            }
            dp_load_slot<false>(a, st, r0, mine + G, n, q, r, unused, wl);  // the next block
            __syncwarp();
            double2 p1 = s_pair[0], p2 = s_pair[1], p3 = s_pair[2], p4 = s_pair[3], w = s_w[0];
            for (int u0 = 0; u0 < G; u0 += UNROLL) {
                const double2* pair_at = s_pair + u0 * NEAR;
#pragma unroll
                for (int v = 0; v < UNROLL; ++v) {
                    const double2 wi = w;
                    const double c4 = __dsub_rn(__dadd_rn(f4, p4.x), p4.y), c3 = __dsub_rn(__dadd_rn(f3, p3.x), p3.y);
                    const double c2 = __dsub_rn(__dadd_rn(f2, p2.x), p2.y), c1 = __dsub_rn(__dadd_rn(f1, p1.x), p1.y);
                    // the next anchor's pairs, ahead of this one's result (the block's last step reads its own again)
                    const int nv = v + 1 < UNROLL || u0 + UNROLL < G ? v + 1 : v;
                    p1 = pair_at[nv * NEAR];
                    p2 = pair_at[nv * NEAR + 1];
                    p3 = pair_at[nv * NEAR + 2];
                    p4 = pair_at[nv * NEAR + 3];
                    w = s_w[u0 + nv];
                    const double x = c4 > wi.x ? c4 : wi.x, y = c2 > c3 ? c2 : c3;
                    const double z = y > x ? y : x;
                    double best = c1 > z ? c1 : z;
                    if (!(older + wi.y < best)) {
                        // an older predecessor may score as much: the rest of the window, oldest first
                        if (gl == 0) ++s_p[G];
                        const int u = u0 + v, i = base + u;
                        const int lim = lb < i ? lb : i;
                        const int2 me = s_qr[i & rm];
                        double bs = 0.0;
                        int ba = 0;
                        for (int t = lim > NEAR ? (lim - NEAR - 1) / G : -1; t >= 0; --t) {
                            const int ag = NEAR + 1 + t * G + gl;
                            if (ag <= lim) {
                                const int2 c = s_qr[(i - ag) & rm];
                                const int dq = me.x - c.x, dr = me.y - c.y;
                                if ((unsigned)(dq - 1) < mg && (unsigned)(dr - 1) < mg) {
                                    const double mn = int_to_double(dq < dr ? dq : dr);
                                    const double sc = __dsub_rn(__dadd_rn(s_f[(i - ag) & rm], mn < wi.x ? mn : wi.x),
                                                                __ldg(&lut[dr > dq ? dr - dq : dq - dr]));
                                    if (sc > wi.x && (ba == 0 || sc > bs)) {
                                        bs = sc;
                                        ba = ag;
                                    }
                                }
                            }
                        }
                        const unsigned gm = G == 32 ? FULL_MASK : ((1u << (G & 31)) - 1u) << (lane & ~(G - 1));
#pragma unroll
                        for (int o = G / 2; o > 0; o >>= 1) {
                            const double os = __shfl_xor_sync(gm, bs, o);
                            const int oa = __shfl_xor_sync(gm, ba, o);
                            if (oa && (ba == 0 || os > bs || (os == bs && oa > ba))) {
                                bs = os;
                                ba = oa;
                            }
                        }
                        if (ba && bs >= best) {
                            best = bs;
                            s_p[u] = ba;
                        }
                    }
                    older = f4 > older && base + u0 + v >= NEAR ? f4 : older;
                    f_at[u0 + v] = best;
                    f4 = f3;
                    f3 = f2;
                    f2 = f1;
                    f1 = best;
                }
            }
            __syncwarp();
            if (mine < n) {
                // the predecessor: an older one, or the oldest near one that gives the score
                const double fi = f_at[gl];
                int age = s_p[gl];
                if (!age && fi > s_w[gl].x) {
#pragma unroll
                    for (int d = 1; d <= NEAR; ++d) {
                        const double2 p = s_pair[gl * NEAR + d - 1];
                        if (__dsub_rn(__dadd_rn(s_f[(mine - d) & rm], p.x), p.y) == fi) age = d;
                    }
                }
                a.f[st + mine] = fi;
                a.parent[st + mine] = age ? mine - age : -1;
            }
            whole = __any_sync(FULL_MASK, s_p[G] >= WHOLE_FROM * G / 32);
        }
    }
}

// ---------------------------------------------------------------------------
// Chain peeling + select: one CTA per read.
// ---------------------------------------------------------------------------
struct PeelArgs {
    int32_t n_reads;
    const int64_t* read_off;
    const int32_t* n_plus;
    const int32_t* n_minus;
    const int32_t* perm;
    const int32_t* read_pos;  // original layout
    const int32_t* ref_pos;
    const int32_t* length;
    const double* f;
    const int32_t* parent;
    int32_t min_chain_anchors;
    int32_t max_chains;
    double min_chain_score;
    double secondary_overlap;
    double secondary_score_ratio;
    // workspace (per anchor, in the read's range)
    unsigned long long* gkey;  // 2 * n_anchors
    int* gidx;                 // 2 * n_anchors
    int32_t* mem_tmp;          // walk members (sorted-local indices), all walks
    double* c_score;           // candidate records; during a strand's walk, c_mem /
    int4* c_span;              // c_span hold every walk's (offset, count) / (start, stop)
    int2* c_mem;               // (member offset within read, count)
    int8_t* c_strand;
    int8_t* claimed;           // per anchor: skipped-start flags, then (strands
                               // beyond the shared buffer) claimed flags
    int smem_elems;
    int64_t cap;               // anchors the workspace arrays hold
    // results
    int32_t* n_chains;
    double* score;
    int32_t* strand;
    int32_t* span;
    int32_t* is_primary;
    int32_t* n_members;
    int32_t* members;
};

// ---------------------------------------------------------------------------
// Reads with one chain.
//
// The first walk of a read starts at the largest f and reaches a root, so its
// score is that f, and no other chain scores more than its own start's f.  Of
// the walks that follow, only those at or above cutoff = best * ratio can be
// selected, and a walk from s stops at the first claimed node above it: on the
// first chain or before, so its score is at most f[s] less the smallest f on
// the way there.  Where that bound stays below the cutoff for every node off
// the chain (and the other strand's largest f does too), the read has one
// chain and nothing else to rank: its members are the ancestors of the start.
//
// They are found without walking them one by one.  Parents precede their
// children, so a warp per block of 32 nodes collects each node's ancestors
// inside the block as a bit mask, and the first ancestor before it, in five
// rounds of doubling; one thread then hops block by block.  A read for which
// the bounds do not hold (several chains above the cutoff, negative scores or
// limits, too few members) is left to the general form below, n_chains = PENDING.
//
// What bounds it is reading f, parents and positions once; the general form
// ranks every possible start and walks them in one thread.  Measured on one
// B200, whole peel: one 15 kb read 264 -> 56 us, 5,000 of them 1,781 ->
// 356 us, 1,000 reads of 10,000 anchors 2,481 -> 398 us.
// ---------------------------------------------------------------------------
constexpr int PENDING = -1;
constexpr int ONE_CAP = 4096, ONE_CAP_BIG = 16384;  // nodes of a strand: 128- and 512-thread blocks
constexpr int ONE_STEPS = 64;                       // nodes between a start and the chain, before giving up

__host__ __device__ constexpr size_t one_smem_bytes(int cap) { return (size_t)cap * 8 + (size_t)cap / 32 * 8; }

template <int T, int CAP>
__device__ void one_chain(const PeelArgs& a, int r, unsigned char* smem) {
    unsigned* s_anc = reinterpret_cast<unsigned*>(smem);                     // in-block ancestors, itself included
    unsigned* s_on = s_anc + CAP;                                            // chain members
    int* s_pre = reinterpret_cast<int*>(s_on + CAP / 32);                    // members before the block
    unsigned short* s_exit = reinterpret_cast<unsigned short*>(s_pre + CAP / 32);  // first ancestor before the block, + 1
    unsigned short* s_par = s_exit + CAP;                                    // parent + 1
    __shared__ double r_max[2][T / 32], r_min[T / 32];
    __shared__ int r_arg[2][T / 32];
    __shared__ int4 r_span[T / 32];
    __shared__ int r_sum[T / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t a0 = a.read_off[r];
    const int np = a.n_plus[r], nm = a.n_minus[r];
    // largest f (first on a tie) per strand, smallest f of both; strands with too few anchors take no part
    const int ns[2] = {np >= a.min_chain_anchors ? np : 0, nm >= a.min_chain_anchors ? nm : 0};
    double mx[2] = {-INFINITY, -INFINITY}, mn = INFINITY;
    int arg[2] = {0x7fffffff, 0x7fffffff};
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const double* f = a.f + a0 + (g ? np : 0);
#pragma unroll 4
        for (int x = tid; x < ns[g]; x += T) {
            const double v = f[x];
            mn = fmin(mn, v);
            if (v > mx[g]) {
                mx[g] = v;
                arg[g] = x;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(FULL_MASK, mx[g], o);
            const int oa = __shfl_xor_sync(FULL_MASK, arg[g], o);
            if (ov > mx[g] || (ov == mx[g] && oa < arg[g])) {
                mx[g] = ov;
                arg[g] = oa;
            }
        }
        if (lane == 0) {
            r_max[g][wid] = mx[g];
            r_arg[g][wid] = arg[g];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(FULL_MASK, mn, o));
    if (lane == 0) r_min[wid] = mn;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < T / 32; ++w) {
        mn = fmin(mn, r_min[w]);
#pragma unroll
        for (int g = 0; g < 2; ++g)
            if (r_max[g][w] > mx[g] || (r_max[g][w] == mx[g] && r_arg[g][w] < arg[g])) {
                mx[g] = r_max[g][w];
                arg[g] = r_arg[g][w];
            }
    }
    const int g = mx[1] > mx[0] ? 1 : 0;  // the first maximum: the plus strand's on a tie
    const double best = mx[g], cutoff = best * a.secondary_score_ratio;
    const int n = g ? nm : np, s0 = g ? np : 0;
    int state = PENDING;
    if (ns[0] == 0 && ns[1] == 0)
        state = 0;
    else if (!(mn >= 0.0) || !(a.secondary_score_ratio >= 0.0) || 0.0 > a.secondary_overlap || n > CAP)
        state = PENDING;  // (an overlap limit below 0 drops the best chain too)
    else if (!(best >= a.min_chain_score))
        state = 0;  // no walk scores more than its start
    else if (ns[1 - g] == 0 || mx[1 - g] < cutoff)
        state = 1;
    if (state != 1) {  // uniform over the block
        if (tid == 0) a.n_chains[r] = state;
        return;
    }
    const double* f = a.f + a0 + s0;
    const int32_t* par = a.parent + a0 + s0;
    const int words = (n + 31) / 32;
    for (int b = wid; b < words; b += T / 32) {
        const int x = 32 * b + lane;
        const int p = x < n ? par[x] : -1;
        int j = p >= 32 * b ? p & 31 : lane;
        unsigned m = 1u << lane;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            m |= __shfl_sync(FULL_MASK, m, j);
            j = __shfl_sync(FULL_MASK, j, j);
        }
        const int out = __shfl_sync(FULL_MASK, p, j);
        s_anc[x] = m;
        s_exit[x] = (unsigned short)(out + 1);
        s_par[x] = (unsigned short)(p + 1);
        if (lane == 0) s_on[b] = 0u;
    }
    __syncthreads();
    if (tid == 0) {
        for (int c = arg[g]; c >= 0;) {
            const unsigned m = s_anc[c];
            const int e = (int)s_exit[c] - 1;
            s_on[c >> 5] = m;
            c = e;
        }
    }
    __syncthreads();
    // every other node of the strand stays below the cutoff
    bool other = false;
    for (int x = tid; x < n; x += T) {
        if ((s_on[x >> 5] >> (x & 31)) & 1u) continue;
        const double fx = f[x];
        if (!(fx >= cutoff)) continue;
        double low = fx;
        int y = x, k = 0;
        do {
            y = (int)s_par[y] - 1;
            low = y >= 0 ? fmin(low, f[y]) : 0.0;
            ++k;
        } while (y >= 0 && !((s_on[y >> 5] >> (y & 31)) & 1u) && k < ONE_STEPS);
        other |= k == ONE_STEPS || fx - low >= cutoff;
    }
    // members before each block, and their number
    int mine = 0;
    constexpr int WPT = CAP / 32 / T > 0 ? CAP / 32 / T : 1;  // blocks per thread
#pragma unroll
    for (int k = 0; k < WPT; ++k) {
        const int b = tid * WPT + k;
        mine += b < words ? __popc(s_on[b]) : 0;
    }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(FULL_MASK, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) r_sum[wid] = incl;
    other = __syncthreads_or(other);
    int at = incl - mine, total = 0;
#pragma unroll
    for (int w = 0; w < T / 32; ++w) {
        at += w < wid ? r_sum[w] : 0;
        total += r_sum[w];
    }
    if (other || total < a.min_chain_anchors) {
        if (tid == 0) a.n_chains[r] = PENDING;
        return;
    }
#pragma unroll
    for (int k = 0; k < WPT; ++k) {
        const int b = tid * WPT + k;
        if (b < words) {
            s_pre[b] = at;
            at += __popc(s_on[b]);
        }
    }
    __syncthreads();
    // members (original indices, read order) and their span
    int rs = 0x7fffffff, re = -0x7fffffff - 1, fs = 0x7fffffff, fe = -0x7fffffff - 1;
#pragma unroll 4
    for (int x = tid; x < n; x += T) {
        const unsigned on = s_on[x >> 5];
        if ((on >> (x & 31)) & 1u) {
            const int o = a.perm[a0 + s0 + x];
            a.members[a0 + s_pre[x >> 5] + __popc(on & ((1u << (x & 31)) - 1u))] = o;
            const int rp = a.read_pos[a0 + o], fp = a.ref_pos[a0 + o], ln = a.length[a0 + o];
            rs = min(rs, rp);
            re = max(re, rp + ln);
            fs = min(fs, fp);
            fe = max(fe, fp + ln);
        }
    }
    rs = __reduce_min_sync(FULL_MASK, rs);
    re = __reduce_max_sync(FULL_MASK, re);
    fs = __reduce_min_sync(FULL_MASK, fs);
    fe = __reduce_max_sync(FULL_MASK, fe);
    if (lane == 0) r_span[wid] = make_int4(rs, re, fs, fe);
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < T / 32; ++w) {
            const int4 q = r_span[w];
            rs = min(rs, q.x);
            re = max(re, q.y);
            fs = min(fs, q.z);
            fe = max(fe, q.w);
        }
        const size_t slot = (size_t)r * a.max_chains;
        a.n_chains[r] = 1;
        a.score[slot] = best;
        a.strand[slot] = g ? -1 : 1;
        a.span[4 * slot + 0] = rs;
        a.span[4 * slot + 1] = re;
        a.span[4 * slot + 2] = fs;
        a.span[4 * slot + 3] = fe;
        a.is_primary[slot] = 1;
        a.n_members[slot] = total;
    }
}

__global__ void __launch_bounds__(128) chain_one_kernel(PeelArgs a) {
    extern __shared__ uint4 one_smem[];
    const int r = blockIdx.x;
    const int np = a.n_plus[r], nm = a.n_minus[r];
    if (a.read_off[r] + np + nm > a.cap) {  // beyond the workspace (the sort reported it): no chains
        if (threadIdx.x == 0) a.n_chains[r] = 0;
        return;
    }
    if (max(np, nm) > ONE_CAP) {  // chain_one_big_kernel
        if (threadIdx.x == 0) a.n_chains[r] = PENDING;
        return;
    }
    one_chain<128, ONE_CAP>(a, r, reinterpret_cast<unsigned char*>(one_smem));
}

// Reads with a strand of more than ONE_CAP anchors: a block looks through
// every gridDim-th read and takes the large ones.
__global__ void __launch_bounds__(512) chain_one_big_kernel(PeelArgs a) {
    extern __shared__ uint4 one_smem[];
    __shared__ int n_found, found[512];
    for (int64_t first = blockIdx.x; first < a.n_reads; first += (int64_t)gridDim.x * 512) {
        if (threadIdx.x == 0) n_found = 0;
        __syncthreads();
        const int64_t r = first + (int64_t)threadIdx.x * gridDim.x;
        if (r < a.n_reads && a.n_chains[r] == PENDING) {
            const int n = max(a.n_plus[r], a.n_minus[r]);
            if (n > ONE_CAP && n <= ONE_CAP_BIG) found[atomicAdd(&n_found, 1)] = (int)r;
        }
        __syncthreads();
        for (int k = 0; k < n_found; ++k) {
            one_chain<512, ONE_CAP_BIG>(a, found[k], reinterpret_cast<unsigned char*>(one_smem));
            __syncthreads();
        }
    }
}

// The general form, for the reads left pending: every walk, ranked and
// selected.
__global__ void __launch_bounds__(128) chain_peel_kernel(PeelArgs a) {
    extern __shared__ unsigned long long pk_smem[];
    const int r = blockIdx.x;
    if (r >= a.n_reads) return;
    const int64_t a0 = a.read_off[r];
    __shared__ int n_cand;
    __shared__ int n_memtot;
    if (threadIdx.x == 0) {
        n_cand = 0;
        n_memtot = 0;
    }
    const int np = a.n_plus[r], nm = a.n_minus[r];
    const int n_sorted = np + nm;
    if (a.n_chains[r] != PENDING) return;
    __shared__ int n_start;
    __shared__ int n_fill;
    __shared__ int n_walk;
    __shared__ int warp_cnt[4];
    for (int seg = 0; seg < 2; ++seg) {
        const int n = seg == 0 ? np : nm;
        const int s0 = seg == 0 ? 0 : np;  // offset of the segment inside the read
        __syncthreads();
        if (n < a.min_chain_anchors || n == 0) continue;
        const double* fs = a.f + a0 + s0;
        const int32_t* par = a.parent + a0 + s0;
        // Walk starts.  A node with a child of higher score is claimed before
        // its own turn (the child ranks first, and the claimed set is closed
        // under predecessors), so the walk skips it in the reference's order:
        // only the other nodes are ranked.  dom[] marks the skipped nodes.
        int8_t* dom = a.claimed + a0;
        for (int x = threadIdx.x; x < n; x += blockDim.x) dom[x] = 0;
        if (threadIdx.x == 0) {
            n_start = 0;
            n_fill = 0;
        }
        __syncthreads();
        for (int x = threadIdx.x; x < n; x += blockDim.x) {
            const int p = par[x];
            if (p >= 0 && fs[x] > fs[p]) dom[p] = 1;
        }
        __syncthreads();
        const int lane = threadIdx.x & 31;
        const unsigned lt = (1u << lane) - 1u;
        for (int x0 = threadIdx.x & ~31; x0 < n; x0 += blockDim.x) {
            const unsigned b = __ballot_sync(FULL_MASK, x0 + lane < n && !dom[x0 + lane]);
            if (lane == 0 && b) atomicAdd(&n_start, __popc(b));
        }
        __syncthreads();
        const int ns = n_start;
        const int np2 = next_pow2(ns);
        unsigned long long* key;
        int* idx;
        // shared buffer of 12 * smem_elems bytes: keys from the bottom, the
        // sorted indices at the top (they outlive the keys: the walk reads them)
        const bool sort_smem = np2 <= a.smem_elems;
        if (sort_smem) {
            key = pk_smem;
            idx = reinterpret_cast<int*>(reinterpret_cast<char*>(pk_smem) + 12 * a.smem_elems - 4 * np2);
        } else {
            key = a.gkey + 2 * a0;  // np2 <= 2n entries of this read's range
            idx = a.gidx + 2 * a0;
        }
        for (int x0 = threadIdx.x & ~31; x0 < n; x0 += blockDim.x) {
            const int x = x0 + lane;
            const bool st = x < n && !dom[x];
            const unsigned b = __ballot_sync(FULL_MASK, st);
            int base = 0;
            if (lane == 0 && b) base = atomicAdd(&n_fill, __popc(b));
            base = __shfl_sync(FULL_MASK, base, 0);
            if (st) {
                // argsort(-f, stable): ascending -f == descending f, ties by index
                const int slot = base + __popc(b & lt);
                key[slot] = ~ordered_bits(fs[x]);
                idx[slot] = x;
            }
        }
        for (int x = ns + threadIdx.x; x < np2; x += blockDim.x) {
            key[x] = ~0ull;
            idx[x] = 0x7fffffff;
        }
        __syncthreads();
        if (sort_smem)
            block_bitonic(pk_smem,
                          reinterpret_cast<int*>(reinterpret_cast<char*>(pk_smem) + 12 * a.smem_elems - 4 * np2),
                          np2);
        else
            block_bitonic(key, idx, np2);
        __syncthreads();
        const int c_first = n_cand;  // chains found in earlier segments
        // The walk is serial in rank order (the reference's loop): one thread
        // takes the starts in order (the next start's index loaded ahead) and
        // walks the unclaimed ones.  Every walk is recorded -- (member offset,
        // count) and (start, stop node) -- and scored afterwards by the whole
        // block.  The strand's walks claim all n nodes, so its members fill
        // mem_tmp[mem_base, mem_base + n).
        const int mem_base = n_memtot;
        if (6 * n + (sort_smem ? 4 * np2 : 0) <= 12 * a.smem_elems) {
            // shared memory, in the dead sort keys below the sorted starts:
            // pw[x] = predecessor + 1 with bit 31 set once claimed (one load
            // per step of a walk), and the member list (16-bit: n <= 4,096)
            int* pw = reinterpret_cast<int*>(pk_smem);
            unsigned short* ml = reinterpret_cast<unsigned short*>(pw + n);
            for (int x = threadIdx.x; x < n; x += blockDim.x) pw[x] = par[x] + 1;
            __syncthreads();
            if (threadIdx.x == 0) {
                int mo = 0, w = c_first;
                int i_next = idx[0];
                for (int k = 0; k < ns; ++k) {
                    const int i = i_next;
                    if (k + 1 < ns) i_next = idx[k + 1];
                    int v = pw[i];
                    if (v < 0) continue;
                    int m = 0;
                    int node = i;
                    do {
                        pw[node] = v | (int)0x80000000u;
                        ml[mo + m] = (unsigned short)node;
                        ++m;
                        node = v - 1;
                        if (node < 0) break;
                        v = pw[node];
                    } while (v >= 0);
                    a.c_mem[a0 + w] = make_int2(mem_base + mo, m);
                    a.c_span[a0 + w] = make_int4(i, node, 0, 0);
                    ++w;
                    mo += m;
                }
                n_walk = w;
            }
            __syncthreads();
            for (int x = threadIdx.x; x < n; x += blockDim.x) a.mem_tmp[a0 + mem_base + x] = (int)ml[x];
        } else {
            int8_t* claimed = a.claimed + a0;  // held the dom flags
            for (int x = threadIdx.x; x < n; x += blockDim.x) claimed[x] = 0;
            __syncthreads();
            if (threadIdx.x == 0) {
                int mo = 0, w = c_first;
                int i_next = idx[0];
                for (int k = 0; k < ns; ++k) {
                    const int i = i_next;
                    if (k + 1 < ns) i_next = idx[k + 1];
                    if (claimed[i]) continue;
                    int m = 0;
                    int node = i;
                    while (node >= 0) {
                        const int8_t cl = claimed[node];
                        const int nx = par[node];
                        if (cl) break;
                        claimed[node] = 1;
                        a.mem_tmp[a0 + mem_base + mo + m] = node;
                        ++m;
                        node = nx;
                    }
                    a.c_mem[a0 + w] = make_int2(mem_base + mo, m);
                    a.c_span[a0 + w] = make_int4(i, node, 0, 0);
                    ++w;
                    mo += m;
                }
                n_walk = w;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) n_memtot = mem_base + n;
        // candidates: the walks with enough members and a partial score
        // f[start] - f[stop] above the floor, kept in walk order (compacted in
        // place, 256 records at a time: a record moves only to a lower slot)
        {
            const int wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
            const int n_w = n_walk;
            for (int w0 = c_first; w0 < n_w; w0 += blockDim.x) {
                const int w = w0 + threadIdx.x;
                bool keep = false;
                double sc = 0.0;
                int2 cm = make_int2(0, 0);
                if (w < n_w) {
                    cm = a.c_mem[a0 + w];
                    const int4 se = a.c_span[a0 + w];
                    sc = fs[se.x] - (se.y >= 0 ? fs[se.y] : 0.0);
                    keep = cm.y >= a.min_chain_anchors && sc >= a.min_chain_score;
                }
                const unsigned kb = __ballot_sync(FULL_MASK, keep);
                if (lane == 0) warp_cnt[wid] = __popc(kb);
                __syncthreads();
                int slot = n_cand + __popc(kb & lt);
                int tot = 0;
                for (int q = 0; q < nwarp; ++q) {
                    if (q < wid) slot += warp_cnt[q];
                    tot += warp_cnt[q];
                }
                __syncthreads();
                if (keep) {
                    a.c_score[a0 + slot] = sc;
                    a.c_mem[a0 + slot] = cm;
                    a.c_strand[a0 + slot] = (int8_t)(seg == 0 ? 1 : -1);
                }
                if (threadIdx.x == 0) n_cand += tot;
                __syncthreads();
            }
        }
        __syncthreads();
    }
    __syncthreads();
    // ---- select ----
    // The reference sorts the candidates by score (stable) and scans them:
    // the first is kept, and once a chain is kept the scan stops at the
    // first score below cutoff = best * ratio.  Only the first maximum and
    // the candidates at or above the cutoff can be visited before that stop
    // (a scan that has kept nothing by then keeps nothing later either), so
    // only they are sorted and only their spans are computed.
    const int nc = n_cand;
    if (nc == 0) {
        if (threadIdx.x == 0) a.n_chains[r] = 0;
        return;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    __shared__ double red_s[4];  // one entry per warp (at most 128 threads)
    __shared__ int red_i[4];
    __shared__ int4 red_span[4];
    {
        double bs = -INFINITY;
        int bi = 0x7fffffff;
        for (int c = threadIdx.x; c < nc; c += blockDim.x) {
            const double sc = a.c_score[a0 + c];
            if (sc > bs || (sc == bs && c < bi)) {
                bs = sc;
                bi = c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double os = __shfl_xor_sync(FULL_MASK, bs, o);
            const int oi = __shfl_xor_sync(FULL_MASK, bi, o);
            if (os > bs || (os == bs && oi < bi)) {
                bs = os;
                bi = oi;
            }
        }
        if (lane == 0) {
            red_s[wid] = bs;
            red_i[wid] = bi;
        }
        if (threadIdx.x == 0) {
            n_start = 0;
            n_fill = 0;
        }
    }
    __syncthreads();
    double best_sc = red_s[0];
    int best_c = red_i[0];
    for (int w = 1; w < nw; ++w) {
        if (red_s[w] > best_sc || (red_s[w] == best_sc && red_i[w] < best_c)) {
            best_sc = red_s[w];
            best_c = red_i[w];
        }
    }
    const double cutoff = best_sc * a.secondary_score_ratio;
    for (int x0 = threadIdx.x & ~31; x0 < nc; x0 += blockDim.x) {
        const int c = x0 + lane;
        const bool in = c < nc && (c == best_c || a.c_score[a0 + c] >= cutoff);
        const unsigned b = __ballot_sync(FULL_MASK, in);
        if (lane == 0 && b) atomicAdd(&n_start, __popc(b));
    }
    __syncthreads();
    const int ns = n_start;
    const int np2 = next_pow2(ns);
    const bool sel_smem = np2 <= a.smem_elems;
    unsigned long long* key;
    int* idx;
    if (sel_smem) {
        key = pk_smem;
        idx = reinterpret_cast<int*>(reinterpret_cast<char*>(pk_smem) + 12 * a.smem_elems - 4 * np2);
    } else {
        key = a.gkey + 2 * a0;
        idx = a.gidx + 2 * a0;
    }
    for (int x0 = threadIdx.x & ~31; x0 < nc; x0 += blockDim.x) {
        const int c = x0 + lane;
        const double sc = c < nc ? a.c_score[a0 + c] : 0.0;
        const bool in = c < nc && (c == best_c || sc >= cutoff);
        const unsigned b = __ballot_sync(FULL_MASK, in);
        int base = 0;
        if (lane == 0 && b) base = atomicAdd(&n_fill, __popc(b));
        base = __shfl_sync(FULL_MASK, base, 0);
        if (in) {
            const int slot = base + __popc(b & lt);
            key[slot] = ~ordered_bits(sc);  // sorted(key=-score), stable
            idx[slot] = c;
        }
    }
    for (int x = ns + threadIdx.x; x < np2; x += blockDim.x) {
        key[x] = ~0ull;
        idx[x] = 0x7fffffff;
    }
    __syncthreads();
    if (sel_smem)
        block_bitonic(pk_smem,
                      reinterpret_cast<int*>(reinterpret_cast<char*>(pk_smem) + 12 * a.smem_elems - 4 * np2),
                      np2);
    else
        block_bitonic(key, idx, np2);
    // spans of the sorted candidates over their members' original
    // coordinates, one candidate at a time across the block
    for (int k = 0; k < ns; ++k) {
        const int c = idx[k];
        const int2 cm = a.c_mem[a0 + c];
        const int s0 = a.c_strand[a0 + c] == 1 ? 0 : np;
        int rs = 0x7fffffff, re = -0x7fffffff - 1, fs = 0x7fffffff, fe = -0x7fffffff - 1;
#pragma unroll 4
        for (int x = threadIdx.x; x < cm.y; x += blockDim.x) {
            const int o = a.perm[a0 + s0 + a.mem_tmp[a0 + cm.x + x]];
            const int rp = a.read_pos[a0 + o], fp = a.ref_pos[a0 + o], ln = a.length[a0 + o];
            rs = min(rs, rp);
            re = max(re, rp + ln);
            fs = min(fs, fp);
            fe = max(fe, fp + ln);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            rs = min(rs, __shfl_xor_sync(FULL_MASK, rs, o));
            re = max(re, __shfl_xor_sync(FULL_MASK, re, o));
            fs = min(fs, __shfl_xor_sync(FULL_MASK, fs, o));
            fe = max(fe, __shfl_xor_sync(FULL_MASK, fe, o));
        }
        if (lane == 0) red_span[wid] = make_int4(rs, re, fs, fe);
        __syncthreads();
        if (threadIdx.x == 0) {
            int4 sp = red_span[0];
            for (int w = 1; w < nw; ++w) {
                const int4 q = red_span[w];
                sp = make_int4(min(sp.x, q.x), max(sp.y, q.y), min(sp.z, q.z), max(sp.w, q.w));
            }
            a.c_span[a0 + c] = sp;
        }
        __syncthreads();
    }
    __shared__ int kept_c[64];
    __shared__ int n_kept;
    if (threadIdx.x == 0) {
        const int mc = a.max_chains < 64 ? a.max_chains : 64;
        int kept = 0;
        for (int k = 0; k < ns; ++k) {
            const int c = idx[k];
            const double sc = a.c_score[a0 + c];
            if (sc < cutoff && kept) break;
            double overlap = 0.0;
            if (kept) {  // only the first kept chain is primary
                const int4 x = a.c_span[a0 + c];
                const int4 y = a.c_span[a0 + kept_c[0]];
                const int lo = max(x.x, y.x), hi = min(x.y, y.y);
                if (hi > lo) {
                    const int den = max(min(x.y - x.x, y.y - y.x), 1);
                    overlap = (double)(hi - lo) / (double)den;
                }
            }
            if (overlap > a.secondary_overlap) continue;
            kept_c[kept++] = c;
            if (kept >= mc) break;
        }
        n_kept = kept;
        a.n_chains[r] = kept;
    }
    __syncthreads();
    // ---- output: records and members (original indices, read order) ----
    int wpos = 0;
    for (int k = 0; k < n_kept; ++k) {
        const int c = kept_c[k];
        const int2 cm = a.c_mem[a0 + c];
        const int s0 = a.c_strand[a0 + c] == 1 ? 0 : np;
        const size_t slot = (size_t)r * a.max_chains + k;
        if (threadIdx.x == 0) {
            a.score[slot] = a.c_score[a0 + c];
            a.strand[slot] = a.c_strand[a0 + c];
            const int4 sp = a.c_span[a0 + c];
            a.span[4 * slot + 0] = sp.x;
            a.span[4 * slot + 1] = sp.y;
            a.span[4 * slot + 2] = sp.z;
            a.span[4 * slot + 3] = sp.w;
            a.is_primary[slot] = k == 0;
            a.n_members[slot] = cm.y;
        }
        // the walk stored members from chain end to start: reverse to read order
        // four members per thread per round: their loads are issued together
        for (int x0 = threadIdx.x; x0 < cm.y; x0 += 4 * blockDim.x) {
            int loc[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int x = x0 + u * blockDim.x;
                loc[u] = x < cm.y ? a.mem_tmp[a0 + cm.x + (cm.y - 1 - x)] : 0;
            }
            int o[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) o[u] = x0 + u * blockDim.x < cm.y ? a.perm[a0 + s0 + loc[u]] : 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int x = x0 + u * blockDim.x;
                if (x < cm.y) a.members[a0 + wpos + x] = o[u];
            }
        }
        wpos += cm.y;
    }
    (void)n_sorted;
}

}  // namespace gmf

using namespace gmf;

namespace {

// Shared-memory sort buffer of the per-strand peel: 2048 keys (24 KB), so 8
// CTAs fit an SM (the peel's serial walk runs in 8 blocks of 4 warps per SM);
// larger strands sort in their own workspace range instead.  The buffer also
// holds a strand's walk state (6 bytes per anchor) beside its sorted starts.
int peel_smem_elems() { return 2048; }

size_t sort_smem_bytes(int elems) { return (size_t)elems * (sizeof(unsigned long long) + sizeof(int)); }

int launch_sort(const gmf_anchor_batch* an, const gmf_sorted_anchors* so, int32_t* len_s, int64_t cap,
                int64_t key_cap, int* err, cudaStream_t stream, const double* lut = nullptr, int max_gap = 0,
                double* min_pen = nullptr) {
    SortArgs s;
    s.lut = lut;
    s.max_gap = max_gap;
    s.min_pen = min_pen;
    s.n_reads = an->n_reads;
    s.read_off = an->read_off;
    s.read_pos = an->read_pos;
    s.ref_pos = an->ref_pos;
    s.length = an->length;
    s.strand = an->strand;
    s.perm = so->perm;
    s.n_plus = so->n_plus;
    s.n_minus = so->n_minus;
    s.read_end_s = so->read_end;
    s.ref_end_s = so->ref_end;
    s.len_s = len_s;
    s.cap = cap;
    s.key_cap = key_cap;
    s.err = err;
    constexpr size_t small = sort_smem_size<256, SORT_CAP>(), big = sort_smem_size<1024, SORT_CAP_BIG>();
    GMF_CUDA_TRY(cudaFuncSetAttribute(chain_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small));
    chain_sort_kernel<<<an->n_reads, 256, small, stream>>>(s);
    GMF_CUDA_TRY(cudaGetLastError());
    if (cap >= 0 && cap <= SORT_CAP) return GMF_OK;  // no read has more
    GMF_CUDA_TRY(cudaFuncSetAttribute(chain_sort_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)big));
    chain_sort_big_kernel<<<std::min(an->n_reads, 148), 1024, big, stream>>>(s);
    return cuda_status(cudaGetLastError());
}

template <int K>
int launch_dp_bcast(const DpArgs& d, int n_segments, cudaStream_t stream) {
    const int wpb = 4;
    const int blocks = (n_segments + wpb - 1) / wpb;
    if (blocks > 0) {
        if (d.weight && d.bonus)
            chain_dp_bcast_kernel<K, true, true><<<blocks, 32 * wpb, 0, stream>>>(d);
        else if (d.weight)
            chain_dp_bcast_kernel<K, true, false><<<blocks, 32 * wpb, 0, stream>>>(d);
        else if (d.bonus)
            chain_dp_bcast_kernel<K, false, true><<<blocks, 32 * wpb, 0, stream>>>(d);
        else
            chain_dp_bcast_kernel<K, false, false><<<blocks, 32 * wpb, 0, stream>>>(d);
    }
    return cuda_status(cudaGetLastError());
}

template <int G>
int launch_dp_near(DpArgs d, int n_segments, cudaStream_t stream) {
    const int lb = d.lookback > 1 ? d.lookback : 1;
    constexpr int GPB = 32 * NEAR_WARPS / G;
    d.ring = next_pow2((lb > NEAR ? lb : NEAR) + G);
    const size_t smem = GPB * near_smem_bytes(G, d.ring);
    GMF_CUDA_TRY(cudaFuncSetAttribute(chain_dp_near_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    const int blocks = (n_segments + GPB - 1) / GPB;
    if (blocks > 0) chain_dp_near_kernel<G><<<blocks, 32 * NEAR_WARPS, smem, stream>>>(d);
    return cuda_status(cudaGetLastError());
}

int launch_dp(DpArgs d, int n_segments, cudaStream_t stream) {
    d.n_segments = n_segments;
    int lb = d.lookback > 1 ? d.lookback : 1;
    // Sorted reads with their lengths as weights: near predecessors first.  A warp for two segments from two
    // long segments per scheduler on (592 on the chip; half the segments are the reads' short strands), if
    // their rings are small.  5,000 reads of 15 kb, whole chain call: 4.19 ms with 32 lanes, 3.87 with 16,
    // 3.96 with 8; 1,000 reads of 75 kb: 5.75, 5.99, 6.80 ms.
    if (d.near) {
        if (n_segments > 2 * 2 * 592 && lb <= 496) return launch_dp_near<16>(d, n_segments, stream);
        return launch_dp_near<32>(d, n_segments, stream);
    }
    // windows up to 224 predecessors: lanes own anchors, K = ceil(lb/32) + 1
    // blocks of 32 in registers
    switch ((lb + 31) / 32 + 1) {
        case 2: return launch_dp_bcast<2>(d, n_segments, stream);
        case 3: return launch_dp_bcast<3>(d, n_segments, stream);
        case 4: return launch_dp_bcast<4>(d, n_segments, stream);
        case 5: return launch_dp_bcast<5>(d, n_segments, stream);
        case 6: return launch_dp_bcast<6>(d, n_segments, stream);
        case 7: return launch_dp_bcast<7>(d, n_segments, stream);
        case 8: return launch_dp_bcast<8>(d, n_segments, stream);
        default: break;
    }
    d.ring = next_pow2(lb + 1);
    const int wpb = 4;
    const size_t smem = (size_t)wpb * d.ring * (sizeof(double) + sizeof(int2));
    GMF_CUDA_TRY(cudaFuncSetAttribute(chain_dp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    const int blocks = (n_segments + wpb - 1) / wpb;
    if (blocks > 0) chain_dp_kernel<<<blocks, 32 * wpb, smem, stream>>>(d);
    return cuda_status(cudaGetLastError());
}

bool valid_lut(const double* lut, int32_t lut_len, int32_t max_gap) {
    return lut != nullptr && lut_len >= max_gap + 1;
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

extern "C" int gmf_chain_dp(int32_t n_rows, const int64_t* row_off, const int32_t* read_end,
                            const int32_t* ref_end, const double* weight, const double* bonus,
                            int32_t max_lookback, int32_t max_gap, const double* pen_lut,
                            int32_t lut_len, double* f, int32_t* parent, gmf_stream_t stream) {
    if (n_rows < 0 || max_gap < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (max_lookback > GMF_MAX_LOOKBACK) return GMF_ERR_LIMIT;
    if (n_rows == 0) return GMF_OK;
    if (!row_off || !read_end || !ref_end || !weight || !f || !parent) return GMF_ERR_INVALID_ARGUMENT;
    if (!valid_lut(pen_lut, lut_len, max_gap)) return GMF_ERR_INVALID_ARGUMENT;
    GMF_BIND_STREAM(stream);
    DpArgs d{};
    d.row_off = row_off;
    d.read_end = read_end;
    d.ref_end = ref_end;
    d.weight = weight;
    d.bonus = bonus;
    d.lookback = max_lookback;
    d.max_gap = max_gap;
    d.lut = pen_lut;
    d.lut_len = lut_len;
    d.f = f;
    d.parent = parent;
    return launch_dp(d, n_rows, (cudaStream_t)stream);
}

extern "C" int gmf_chain_sort(const gmf_anchor_batch* an, const gmf_sorted_anchors* so,
                              void* workspace, size_t workspace_bytes, gmf_stream_t stream) {
    if (!an || !so || an->n_reads < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (an->n_reads == 0) return GMF_OK;
    if (!an->read_off || !an->read_pos || !an->ref_pos || !an->length || !an->strand ||
        !so->perm || !so->n_plus || !so->n_minus || !so->read_end || !so->ref_end)
        return GMF_ERR_INVALID_ARGUMENT;
    if (!workspace || workspace_bytes < 256) return GMF_ERR_WORKSPACE;
    GMF_BIND_STREAM(stream);
    // reads of more than SORT_CAP anchors are sorted when the workspace has 12 * 2 bytes per anchor up to
    // theirs (gmf_chain_workspace_bytes covers it)
    const size_t A = (workspace_bytes - 256) / 24;
    char* p = (char*)workspace;
    int* err = (int*)p;
    const bool fits = 256 + align256(2 * A * 8) + 2 * A * 4 <= workspace_bytes;
    GMF_CUDA_TRY(cudaMemsetAsync(err, 0, 4, (cudaStream_t)stream));
    return launch_sort(an, so, nullptr, -1, fits ? (int64_t)A : 0, err, (cudaStream_t)stream);
}

extern "C" size_t gmf_chain_workspace_bytes(int32_t n_reads, int64_t n_anchors) {
    const size_t A = (size_t)(n_anchors > 0 ? n_anchors : 0);
    const size_t R = (size_t)(n_reads > 0 ? n_reads : 0);
    size_t b = 256;                       // error word
    b += align256(2 * A * 8);             // gkey
    b += align256(2 * A * 4);             // gidx
    b += align256(A * 4) * 3;             // perm, read_end_s, ref_end_s
    b += align256(R * 4) * 2;             // n_plus, n_minus
    b += align256(A * 8);                 // f
    b += align256(A * 4);                 // parent
    b += align256(A * 4);                 // mem_tmp
    b += align256(A * 8);                 // c_score
    b += align256(A * 16);                // c_span
    b += align256(A * 8);                 // c_mem
    b += align256(2 * A);                 // c_strand + claimed flags
    return b;
}

extern "C" int gmf_chain_batch(const gmf_anchor_batch* an, const gmf_chain_params* cp,
                               const double* pen_lut, int32_t lut_len,
                               const gmf_sorted_anchors* sorted_in, const double* sorted_weight,
                               const double* sorted_bonus, const gmf_chain_results* res,
                               void* workspace, size_t workspace_bytes, gmf_stream_t stream_) {
    const cudaStream_t stream = (cudaStream_t)stream_;
    if (!an || !cp || !res || an->n_reads < 0) return GMF_ERR_INVALID_ARGUMENT;
    if (cp->max_lookback > GMF_MAX_LOOKBACK) return GMF_ERR_LIMIT;
    if (cp->max_gap < 0 || cp->max_chains < 1 || cp->max_chains > 64) return GMF_ERR_INVALID_ARGUMENT;
    if (an->n_reads == 0) return GMF_OK;
    if (!an->read_off || !an->read_pos || !an->ref_pos || !an->length || !an->strand)
        return GMF_ERR_INVALID_ARGUMENT;
    if (!res->n_chains || !res->score || !res->strand || !res->span || !res->is_primary ||
        !res->n_members || !res->members)
        return GMF_ERR_INVALID_ARGUMENT;
    if (!valid_lut(pen_lut, lut_len, cp->max_gap)) return GMF_ERR_INVALID_ARGUMENT;
    if ((sorted_weight || sorted_bonus) && !sorted_in) return GMF_ERR_INVALID_ARGUMENT;
    if (!workspace) return GMF_ERR_WORKSPACE;
    GMF_BIND_STREAM(stream);

    // the host does not know n_anchors (device CSR); the caller sized the
    // workspace with gmf_chain_workspace_bytes, so derive A from its size.
    // Layout is computed for the largest A that fits.
    const size_t R = (size_t)an->n_reads;
    size_t lo = 0, hi = workspace_bytes;
    while (lo < hi) {  // largest A with bytes(R, A) <= workspace_bytes
        const size_t mid = (lo + hi + 1) / 2;
        if (gmf_chain_workspace_bytes((int32_t)R, (int64_t)mid) <= workspace_bytes)
            lo = mid;
        else
            hi = mid - 1;
    }
    const size_t A = lo;
    char* p = (char*)workspace;
    int* err = (int*)p;
    p += 256;
    auto take = [&](size_t bytes) {
        char* q = p;
        p += align256(bytes);
        return q;
    };
    unsigned long long* gkey = (unsigned long long*)take(2 * A * 8);
    int* gidx = (int*)take(2 * A * 4);
    gmf_sorted_anchors so;
    int32_t* perm_w = (int32_t*)take(A * 4);
    int32_t* re_w = (int32_t*)take(A * 4);
    int32_t* fe_w = (int32_t*)take(A * 4);
    int32_t* npl_w = (int32_t*)take(R * 4);
    int32_t* nmi_w = (int32_t*)take(R * 4);
    double* f = (double*)take(A * 8);
    int32_t* parent = (int32_t*)take(A * 4);
    int32_t* mem_tmp = (int32_t*)take(A * 4);
    double* c_score = (double*)take(A * 8);
    int4* c_span = (int4*)take(A * 16);
    int2* c_mem = (int2*)take(A * 8);
    int8_t* c_strand = (int8_t*)take(2 * A);
    if (sorted_in) {
        so = *sorted_in;
    } else {
        so.perm = perm_w;
        so.n_plus = npl_w;
        so.n_minus = nmi_w;
        so.read_end = re_w;
        so.ref_end = fe_w;
    }
    GMF_CUDA_TRY(cudaMemsetAsync(err, 0, 256, stream));
    int st;
    const bool near = !sorted_in && cp->max_gap <= NEAR_MAX_GAP;
    double* min_pen = near ? (double*)(err + 2) : nullptr;  // behind the error word
    if (!sorted_in) {
        st = launch_sort(an, &so, mem_tmp, (int64_t)A, (int64_t)A, err, stream, pen_lut, cp->max_gap, min_pen);
        if (st) return st;
    }
    DpArgs d{};
    d.read_off = an->read_off;
    d.n_plus = so.n_plus;
    d.n_minus = so.n_minus;
    d.read_end = so.read_end;
    d.ref_end = so.ref_end;
    d.weight = sorted_weight;
    d.length = an->length;
    d.len_s = sorted_in ? nullptr : mem_tmp;  // the sort left them where the peel will keep its members
    d.perm = so.perm;
    d.bonus = sorted_bonus;
    d.lookback = cp->max_lookback;
    d.max_gap = cp->max_gap;
    d.lut = pen_lut;
    d.lut_len = lut_len;
    d.f = f;
    d.parent = parent;
    d.cap = (int64_t)A;
    d.near = near;
    d.min_pen = min_pen;
    st = launch_dp(d, 2 * an->n_reads, stream);
    if (st) return st;

    PeelArgs k{};
    k.n_reads = an->n_reads;
    k.read_off = an->read_off;
    k.n_plus = so.n_plus;
    k.n_minus = so.n_minus;
    k.perm = so.perm;
    k.read_pos = an->read_pos;
    k.ref_pos = an->ref_pos;
    k.length = an->length;
    k.f = f;
    k.parent = parent;
    k.min_chain_anchors = cp->min_chain_anchors;
    k.max_chains = cp->max_chains;
    k.min_chain_score = cp->min_chain_score;
    k.secondary_overlap = cp->secondary_overlap;
    k.secondary_score_ratio = cp->secondary_score_ratio;
    k.gkey = gkey;
    k.gidx = gidx;
    k.mem_tmp = mem_tmp;
    k.c_score = c_score;
    k.c_span = c_span;
    k.c_mem = c_mem;
    k.c_strand = c_strand;
    k.claimed = c_strand + A;
    k.smem_elems = peel_smem_elems();
    k.cap = (int64_t)A;
    k.n_chains = res->n_chains;
    k.score = res->score;
    k.strand = res->strand;
    k.span = res->span;
    k.is_primary = res->is_primary;
    k.n_members = res->n_members;
    k.members = res->members;
    GMF_CUDA_TRY(cudaFuncSetAttribute(chain_one_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)one_smem_bytes(ONE_CAP)));
    chain_one_kernel<<<an->n_reads, 128, one_smem_bytes(ONE_CAP), stream>>>(k);
    GMF_CUDA_TRY(cudaGetLastError());
    if (A > (size_t)ONE_CAP) {  // a strand may have more
        GMF_CUDA_TRY(cudaFuncSetAttribute(chain_one_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)one_smem_bytes(ONE_CAP_BIG)));
        chain_one_big_kernel<<<std::min(an->n_reads, 148), 512, one_smem_bytes(ONE_CAP_BIG), stream>>>(k);
        GMF_CUDA_TRY(cudaGetLastError());
    }
    const size_t smem = sort_smem_bytes(k.smem_elems);
    GMF_CUDA_TRY(cudaFuncSetAttribute(chain_peel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    chain_peel_kernel<<<an->n_reads, 128, smem, stream>>>(k);
    return cuda_status(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Allocation-free chaining: the scratch is a fixed array of this library.
// ---------------------------------------------------------------------------

// Scratch of gmf_chain_batch_noalloc, one copy per GPU that loads the library.
// Host code must not pass `g_chain_scratch` itself to a kernel (on the host it
// names a stand-in, not device memory); it uses the address looked up below.
static __device__ __align__(256) unsigned char g_chain_scratch[GMF_CHAIN_NOALLOC_SCRATCH_BYTES];

namespace {

constexpr int kMaxScratchDevices = 64;
std::mutex g_scratch_mu;
void* g_scratch_addr[kMaxScratchDevices] = {};

// Device address of g_chain_scratch on the current device, looked up once per
// device (the lookup may load this library's module on that device).
int chain_scratch_address(void** out) {
    int dev = 0;
    GMF_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxScratchDevices) return GMF_ERR_LIMIT;
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_chain_scratch);
        if (e != cudaSuccess || !p) return GMF_ERR_CUDA;
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return GMF_OK;
}

}  // namespace

extern "C" int gmf_chain_batch_noalloc(const gmf_anchor_batch* an, const gmf_chain_params* cp,
                                       const double* pen_lut, int32_t lut_len, int64_t n_anchors,
                                       const gmf_chain_results* res, gmf_stream_t stream) {
    if (!an || !cp || !res || an->n_reads < 0 || n_anchors < 0) return GMF_ERR_INVALID_ARGUMENT;
    const size_t need = gmf_chain_workspace_bytes(an->n_reads, n_anchors);
    if (need > GMF_CHAIN_NOALLOC_SCRATCH_BYTES) return GMF_ERR_LIMIT;
    if (an->n_reads == 0) return GMF_OK;
    GMF_BIND_STREAM(stream);
    void* scratch = nullptr;
    GMF_TRY(chain_scratch_address(&scratch));
    // gmf_chain_batch clears the error word itself; every other scratch array
    // is written before it is read (sort keys, DP values, claimed flags)
    return gmf_chain_batch(an, cp, pen_lut, lut_len, nullptr, nullptr, nullptr, res, scratch, need,
                           stream);
}

extern "C" int gmf_chain_noalloc_error_flags(int32_t* flags, gmf_stream_t stream) {
    if (!flags) return GMF_ERR_INVALID_ARGUMENT;
    GMF_BIND_STREAM(stream);
    void* scratch = nullptr;
    GMF_TRY(chain_scratch_address(&scratch));
    // the error word is the first word of the scratch (gmf_chain_batch's layout)
    return cuda_status(cudaMemcpyAsync(flags, scratch, sizeof(int32_t), cudaMemcpyDefault, (cudaStream_t)stream));
}
