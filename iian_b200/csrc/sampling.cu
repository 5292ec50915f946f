// Sampling over float32 logits rows on the device: greedy argmax and temperature sampling with
// min-p, top-k and top-p truncation.
//
// Semantics follow the reference's CPU sampler (src/iian/sampler.cpp:111-171):
//  * temperature < 1e-5 -> greedy; ties resolve to the lowest id (src/iian/vec_math.h:78-82);
//  * else z = logit / T; min_p keeps z >= max(z) + log(min_p) (:122-126); top_k keeps the k largest
//    with (value desc, id asc) order, only if k is smaller than the candidate count (:131-134);
//    probabilities are exp(z - max) normalised over the candidates (:139-156); top_p keeps the
//    shortest prefix in that order whose mass reaches top_p (:158-163); a uniform draw over the kept
//    mass picks the token by walking the candidates and subtracting (:165-171).
// Differences: the walk is in vocabulary order for every setting (the reference walks in sorted
// order when it sorted), and the uniform number comes from the caller (a counter-based stream per
// request) instead of a per-request mt19937_64.  The distribution is the same.
//
// The k-th largest value and the top-p cut are found exactly, over the order-preserving integer image of the float values.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace iian {

constexpr int kSampleThreads = 1024;

__device__ __forceinline__ unsigned order_key(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// (max value, lowest index holding it) over a row
__device__ __forceinline__ void block_argmax(const float * row, int V, float scale, float & best, int & best_idx,
                                             float * fs, int * is) {
    float b = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float v = row[i] * scale;
        if (v > b || (v == b && i < bi)) { b = v; bi = i; }   // NaN compares false: treated as smaller
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, b, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) { fs[warp] = b; is[warp] = bi; }
    __syncthreads();
    b = lane < (blockDim.x >> 5) ? fs[lane] : -INFINITY;
    bi = lane < (blockDim.x >> 5) ? is[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, b, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
    }
    best = b;
    best_idx = bi == 0x7fffffff ? 0 : bi;
}

__global__ void __launch_bounds__(kSampleThreads) argmax_kernel(const float * __restrict__ logits, int V, size_t stride,
                                                                int * __restrict__ out) {
    __shared__ float fs[32];
    __shared__ int is[32];
    float b; int bi;
    block_argmax(logits + (size_t) blockIdx.x * stride, V, 1.0f, b, bi, fs, is);
    if (threadIdx.x == 0) out[blockIdx.x] = bi;
}

// Two-stage argmax for wide rows: `parts` blocks per row each reduce a contiguous slice to (value, id),
// a second launch reduces the parts.  Ties still go to the lowest id.
__global__ void __launch_bounds__(256) argmax_partial_kernel(const float * __restrict__ logits, int V, size_t stride,
                                                             int parts, float * __restrict__ part_val,
                                                             int * __restrict__ part_idx) {
    __shared__ float fs[32];
    __shared__ int is[32];
    pdl_wait();
    pdl_launch_dependents();
    const int row = blockIdx.y, part = blockIdx.x;
    const int per = (V + parts - 1) / parts;
    const int begin = min(V, part * per), end = min(V, begin + per);
    const float * r = logits + (size_t) row * stride;
    float b = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const float v = r[i];
        if (v > b || (v == b && i < bi)) { b = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, b, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { fs[warp] = b; is[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        b = lane < (blockDim.x >> 5) ? fs[lane] : -INFINITY;
        bi = lane < (blockDim.x >> 5) ? is[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, b, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
        }
        if (lane == 0) { part_val[(size_t) row * parts + part] = b; part_idx[(size_t) row * parts + part] = bi; }
    }
}

__global__ void argmax_final_kernel(const float * __restrict__ part_val, const int * __restrict__ part_idx, int parts,
                                    int * __restrict__ out) {
    pdl_wait();
    pdl_launch_dependents();
    const int row = blockIdx.x, lane = threadIdx.x;       // one warp per row
    float b = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = lane; i < parts; i += 32) {
        const float v = part_val[(size_t) row * parts + i];
        const int idx = part_idx[(size_t) row * parts + i];
        if (v > b || (v == b && idx < bi)) { b = v; bi = idx; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, b, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
    }
    if (lane == 0) out[row] = bi == 0x7fffffff ? 0 : bi;
}

// ---- temperature sampling ------------------------------------------------------------------------------------------
// A row is worked on by a thread-block cluster: each CTA keeps a slice of the row in shared memory as ordered integer keys,
// so the row is read from global memory once (V > 8 x kStagedMax: read again per pass) and a row of 150,000 entries has up
// to 8 SMs.  The k-th largest value and the top-p cut are found exactly.
//  * top-k up to half the cluster's warps: the entries not below the k-th largest of the warps' largest values are listed -- a few more
//    than k --, every CTA takes over all lists, sorts and draws from them, and the row is not scanned again (draw_from_list).
//  * Else the candidates fall into bins by their distance from the largest value (counts, or for top-p masses as integers, so that no
//    order of adding matters), the CTAs add the cluster's bins up, and the entries of the bin that holds the cut are listed (cut_by_bins).
//  * Where more than kListMax entries would be listed (a row of 151,936 with T = 1.0 and top-p 0.95 does that as a rule, and so do many equal
//    logits), the interval of keys that belongs to the cut's bin is narrowed eight ways per pass, and all keys' where the cut lies in the last, open
//    bin: a pass counts (and for top-p adds the probability of) the keys at or above seven borders inside the interval, and the CTAs swap their
//    numbers through each other's shared memory behind one cluster barrier.
// Every sum has an order fixed by V alone (entries of a thread, lanes, warps, CTAs), or is one of integers: the same row gives the same token
// whatever else is in the batch.
// What bounds it: latency -- the row's way in (4 us), three scans of a slice (bins 6.5, list 3, draw 4.5 us) and the barriers between them --
// and two waves of CTAs from 38 rows on.  Rows of 151,936, the usual mix of settings, caches flushed: 48 rows 53 us, 8 rows 38 us, one row with
// top-k and top-p 18 us (by narrowing alone, some 20 passes, caches warm: 123, 82 and 51 us).
constexpr int kDrawThreads = 512;
constexpr int kDrawWarps = kDrawThreads / 32;
constexpr int kDrawCluster = 8;                  // CTAs per row, at most
static_assert(kDrawWarps == 16, "lists are merged by two warps for each CTA");
constexpr int kSliceGoal = 13000;                // entries of a slice before a row gets more CTAs
// Entries a thread asks for before it uses the first: a slice in one trip to memory, and a short remainder not entry by entry (rows of 50,257, one
// with plain temperature 21.5 -> 18, 48 of the usual mix 33.8 -> 31.7; 48 of 151,936 57.2 -> 53.3).
constexpr int kAsked = kSliceGoal / kDrawThreads;
constexpr int kStagedMax = 50 * 1024;            // entries of a slice that shared memory holds (200 KB)
constexpr int kBorders = 7;
constexpr int kBins = kDrawThreads;              // a thread per bin, the last one open
constexpr int kListMax = 1024;                   // entries that are sorted, two a thread

// Bins by the distance from the largest value, 16 to a halving of the mass.  Masses of a bin are whole multiples of 2^-bin_bits: a mass lies
// above half of 2^-(bin / 16) (up to rounding), so its last bit is worth at least 2^-bin_bits times two, and the multiple is at most 2^25.  What
// falls into the last, open bin is cut off below that.
constexpr float kBinsPerUnit = 16.0f * 1.4426950409f;
__device__ __forceinline__ int bin_bits(int bin) { return 25 + (bin >> 4); }

// NaN: below every key that is looked at; the two zeros are equal values and get one key
__device__ __forceinline__ unsigned draw_key(float z) { return z != z ? 0u : order_key(z + 0.0f); }
__device__ __forceinline__ float key_value(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

struct DrawShared {
    double inbox_m[2][kDrawCluster][8];          // what every CTA of the cluster sent: masses (or a value of the kind at hand)
    int inbox_c[2][kDrawCluster][8];             // and counts
    float warp_m[kDrawWarps][8];
    int warp_c[kDrawWarps][8];
    double warp_d[kDrawWarps];
    int warp_i[kDrawWarps];
    int pick;
    int n_list, found[2], n_span, c_above, c_at;
    double m_above, m_at, target;                // with found[0], the cut's bin: masses and counts in front of it and with it, the mass to reach
    unsigned long long warp_q[kDrawWarps];
    unsigned lo_key, hi_key;
    float tops[kDrawCluster * kDrawWarps];       // the largest value of every warp of the cluster
    unsigned long long list[kListMax];           // this CTA's entries that take part in the sort: key, then ~id
    union {                                      // the bins have been read by all before any CTA sorts
        struct { int count[kBins]; unsigned low[kBins], high[kBins]; } bins;     // the masses' last 13 bits and the rest
        unsigned long long sorted[kListMax];
    };
};

template <bool STAGED>
struct Draw {
    DrawShared & sh;
    const unsigned * keys;                       // staged slice
    const float * slice;                         // the same entries in global memory
    int n;                                       // entries of this CTA
    float inv_t, zmax;
    int rank, ctas, turn;
    __device__ __forceinline__ unsigned key(int i) const { return STAGED ? keys[i] : draw_key(slice[i] * inv_t); }
    __device__ __forceinline__ float mass(unsigned k) const { return expf(key_value(k) - zmax); }

    // Lane j of every warp gets (count, mass) of the keys in [max(border j, lo), hi) over the whole row, j < 7; border in lane j.
    template <bool MASS>
    __device__ __forceinline__ void pass(unsigned border, unsigned lo, unsigned hi, int & count, double & m) {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        unsigned t[kBorders];
#pragma unroll
        for (int j = 0; j < kBorders; j++) t[j] = __shfl_sync(0xffffffffu, border, j);
        int c[kBorders];
        float a[8];
#pragma unroll
        for (int j = 0; j < 8; j++) { a[j] = 0.0f; if (j < kBorders) c[j] = 0; }
        for (int i = tid; i < n; i += kDrawThreads) {
            const unsigned k = key(i);
            if (k >= lo && k < hi) {
                const float e = MASS ? mass(k) : 0.0f;
#pragma unroll
                for (int j = 0; j < kBorders; j++) {
                    const bool in = k >= t[j];
                    c[j] += in;
                    if (MASS) a[j] += in ? e : 0.0f;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kBorders; j++) c[j] = __reduce_add_sync(0xffffffffu, c[j]);
        if (MASS) {
            // eight sums over 32 lanes: halve the values a lane carries with every exchange; lane ends with value lane >> 2
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool up = lane & 16;
                const float give = up ? a[j] : a[j + 4], keep = up ? a[j + 4] : a[j];
                a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const bool up = lane & 8;
                const float give = up ? a[j] : a[j + 2], keep = up ? a[j + 2] : a[j];
                a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
            {
                const bool up = lane & 4;
                const float give = up ? a[0] : a[1], keep = up ? a[1] : a[0];
                a[0] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
            }
            a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
            a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
            if ((lane & 3) == 0) sh.warp_m[warp][lane >> 2] = a[0];
        }
        if (lane == 0) {
#pragma unroll
            for (int j = 0; j < kBorders; j++) sh.warp_c[warp][j] = c[j];
        }
        __syncthreads();
        if (warp < kBorders) {                   // warp j puts border j's numbers together and sends them to every CTA
            const int w = lane & (kDrawWarps - 1);
            double d = MASS && lane < kDrawWarps ? (double) sh.warp_m[w][warp] : 0.0;
            const int cc = __reduce_add_sync(0xffffffffu, lane < kDrawWarps ? sh.warp_c[w][warp] : 0);
            if (MASS) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            }
            send(lane, warp, d, cc);
        }
        swap();
        count = 0;
        m = 0.0;
        if (lane < kBorders) {
            for (int r = 0; r < ctas; r++) {
                count += sh.inbox_c[turn][r][lane];
                if (MASS) m += sh.inbox_m[turn][r][lane];
            }
        }
        turn ^= 1;
    }
    // lane r < ctas: value `which` of this CTA goes to CTA r
    __device__ __forceinline__ void send(int lane, int which, double d, int c) {
        if (lane < ctas) {
            cg::cluster_group cl = cg::this_cluster();
            DrawShared * to = cl.map_shared_rank(&sh, lane);
            to->inbox_m[turn][rank][which] = d;
            to->inbox_c[turn][rank][which] = c;
        }
    }
    // what was sent before is there afterwards.  The two inboxes take turns: one is written again only behind the barrier of
    // the turn between, which a CTA reaches after it has read this one.
    __device__ __forceinline__ void swap() { cg::this_cluster().sync(); }

    // The largest key K in [lo, hi) whose count (or mass) of keys at or above it reaches the goal; it does at lo and does not at hi.
    // In: the aggregates at lo and hi; whether the interval may be all keys.  Out: lo = K and the aggregates of the keys at or above it and above it.
    template <bool MASS>
    __device__ __forceinline__ void search(unsigned & lo, unsigned hi, int & c_lo, int & c_hi, double & m_hi, double goal, bool first) {
        const int lane = threadIdx.x & 31;
        while (hi - lo > 1) {
            if (c_lo - c_hi == 1) {              // one key left inside: it is K
                unsigned found = 0;
                for (int i = threadIdx.x; i < n; i += kDrawThreads) {
                    const unsigned k = key(i);
                    if (k >= lo && k < hi) found = k;
                }
                found = __reduce_max_sync(0xffffffffu, found);
                if (lane == 0) sh.warp_i[threadIdx.x >> 5] = (int) found;
                __syncthreads();
                if (threadIdx.x < 32) {
                    found = __reduce_max_sync(0xffffffffu, lane < kDrawWarps ? (unsigned) sh.warp_i[lane] : 0u);
                    send(lane, 0, 0.0, (int) found);
                }
                swap();
                found = __reduce_max_sync(0xffffffffu, lane < ctas ? (unsigned) sh.inbox_c[turn][lane][0] : 0u);
                turn ^= 1;
                lo = found;
                return;
            }
            unsigned border;
            if (first) {                         // distances from the largest value: 32, 16, ..., 0.5
                border = order_key(zmax - exp2f((float) (5 - min(lane, kBorders - 1))));
                border = min(max(border, lo), hi);
            } else border = lo + (unsigned) (((unsigned long long) (hi - lo) * (unsigned) (min(lane, kBorders - 1) + 1)) >> 3);
            first = false;
            int c;
            double m;
            pass<MASS>(border, lo, hi, c, m);
            c += c_hi;
            m += m_hi;
            const unsigned ok = __ballot_sync(0xffffffffu, lane < kBorders && (MASS ? m >= goal : (double) c >= goal));
            const int reached = __popc(ok);      // the borders ascend: the first `reached` of them reach the goal
            const int up = min(reached, kBorders - 1), down = max(reached - 1, 0);
            const unsigned b_up = __shfl_sync(0xffffffffu, border, up), b_down = __shfl_sync(0xffffffffu, border, down);
            const int c_up = __shfl_sync(0xffffffffu, c, up), c_down = __shfl_sync(0xffffffffu, c, down);
            const double m_up = __shfl_sync(0xffffffffu, m, up);
            if (reached < kBorders) { hi = b_up; c_hi = c_up; m_hi = m_up; }
            if (reached > 0) { lo = b_down; c_lo = c_down; }
        }
    }
};

// Sums from the first thread to this one (inclusive), in an order fixed by the block: `total` is everyone's.
__device__ __forceinline__ void block_scan(DrawShared & sh, int & c, double & m, int & c_total, double & m_total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int cv = __shfl_up_sync(0xffffffffu, c, o);
        const double mv = __shfl_up_sync(0xffffffffu, m, o);
        if (lane >= o) { c += cv; m += mv; }
    }
    __syncthreads();
    if (lane == 31) { sh.warp_i[warp] = c; sh.warp_d[warp] = m; }
    __syncthreads();
    int c_before = 0;
    double m_before = 0.0;
    c_total = 0;
    m_total = 0.0;
    for (int w = 0; w < kDrawWarps; w++) {
        if (w == warp) { c_before = c_total; m_before = m_total; }
        c_total += sh.warp_i[w];
        m_total += sh.warp_d[w];
    }
    c += c_before;
    m += m_before;
}

// sh.sorted[0, n) in falling order, no two alike: an entry's place is the number of larger ones, which costs less than a sort for the
// few dozen that are left as a rule (a bitonic one of 30 entries 4,800 clocks, of 500 15,000).
__device__ __forceinline__ void block_sort(DrawShared & sh, int n) {
    unsigned long long v[2];
    int place[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 2; e++) v[e] = (int) threadIdx.x + e * kDrawThreads < n ? sh.sorted[threadIdx.x + e * kDrawThreads] : 0ull;
    if (threadIdx.x < n) {
#pragma unroll 4
        for (int i = 0; i < n; i++) {
            const unsigned long long other = sh.sorted[i];
            place[0] += other > v[0];
            place[1] += other > v[1];
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; e++)
        if ((int) threadIdx.x + e * kDrawThreads < n) sh.sorted[place[e]] = v[e];
    __syncthreads();
}

// The lists of all CTAs, in no order, in every CTA's sh.sorted.  Returns how many; above kListMax nothing is there.
template <bool STAGED>
__device__ __forceinline__ int merge_lists(const Draw<STAGED> & d) {
    cg::cluster_group cl = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    cl.sync();
    // counts: a lane per CTA; entries: two warps per CTA (kDrawWarps = 2 x kDrawCluster)
    const int own = lane < d.ctas ? cl.map_shared_rank(&d.sh, lane)->n_list : 0;
    const int n = __reduce_add_sync(0xffffffffu, own);
    if (n > kListMax) return n;
    const int r = warp >> 1, of_r = __shfl_sync(0xffffffffu, own, r), at = __reduce_add_sync(0xffffffffu, lane < r ? own : 0);
    if (r < d.ctas) {
        const DrawShared * from = cl.map_shared_rank(&d.sh, r);
        for (int i = (warp & 1) * 32 + lane; i < of_r; i += 64) d.sh.sorted[at + i] = from->list[i];
    }
    __syncthreads();
    return n;
}

// The shortest run of the sorted list that reaches `share` of its first `limit` entries' mass.
template <bool STAGED>
__device__ __forceinline__ int shortest_run(const Draw<STAGED> & d, int limit, float share) {
    DrawShared & sh = d.sh;
    const int tid = threadIdx.x;
    double own[2], run, in_list;
#pragma unroll
    for (int e = 0; e < 2; e++) own[e] = 2 * tid + e < limit ? (double) d.mass((unsigned) (sh.sorted[2 * tid + e] >> 32)) : 0.0;
    run = own[0] + own[1];
    int none = 0, none_total;
    block_scan(sh, none, run, none_total, in_list);
    const double goal = (double) share * in_list;
    if (tid == 0) sh.found[1] = limit;
    __syncthreads();
    if (2 * tid + 1 < limit && run >= goal) atomicMin(&sh.found[1], 2 * tid + 2);
    if (2 * tid < limit && run - own[1] >= goal) atomicMin(&sh.found[1], 2 * tid + 1);
    __syncthreads();
    return sh.found[1];
}

// A row with top-k of which few entries are left: they are listed, sorted and drawn from, without another scan.  What bounds the list
// from below is the k-th largest of the warps' largest values: k entries at least are as large.  False: too many, nothing drawn.
template <bool STAGED>
__device__ __forceinline__ bool draw_from_list(const Draw<STAGED> & d, int begin, int k, float P, unsigned cut, float uniform, int & token) {
    DrawShared & sh = d.sh;
    const int tid = threadIdx.x, tops = d.ctas * kDrawWarps;
    if (tid == 0) { sh.n_list = 0; sh.found[0] = kListMax; }
    __syncthreads();
    if (tid < tops) {                            // this warp's rank among them, equal ones by place
        const float own = sh.tops[tid];
        int rank = 0;
#pragma unroll 8
        for (int i = 0; i < tops; i++) rank += sh.tops[i] > own || (sh.tops[i] == own && i < tid);
        if (rank == k - 1) sh.n_span = (int) draw_key(own);
    }
    __syncthreads();
    const unsigned least = max(cut, (unsigned) sh.n_span);
#pragma unroll 4
    for (int i = tid; i < d.n; i += kDrawThreads) {
        const unsigned key = d.key(i);
        if (key < least) continue;
        const int at = atomicAdd(&sh.n_list, 1);
        if (at < kListMax) sh.list[at] = ((unsigned long long) key << 32) | (0xffffffffu - (unsigned) (begin + i));
    }
    const int n = merge_lists(d);
    if (n > kListMax) return false;
    block_sort(sh, n);                           // largest first, equal values by id
    int kept = min(k, n);
    if (P < 1.0f) kept = shortest_run(d, kept, P);
    unsigned long long mine[2];                  // in the vocabulary's order
#pragma unroll
    for (int e = 0; e < 2; e++) mine[e] = 2 * tid + e < kept ? sh.sorted[2 * tid + e] : 0ull;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; e++)
        if (2 * tid + e < kept) sh.sorted[2 * tid + e] = mine[e] << 32 | mine[e] >> 32;
    __syncthreads();
    block_sort(sh, kept);
    double own[2], run, total;
#pragma unroll
    for (int e = 0; e < 2; e++) own[e] = 2 * tid + e < kept ? (double) d.mass((unsigned) sh.sorted[2 * tid + e]) : 0.0;
    run = own[0] + own[1];
    int none = 0, none_total;
    if (tid == 0) sh.found[1] = 0;
    block_scan(sh, none, run, none_total, total);
    const double u = (double) uniform * total;
    if (own[0] > 0.0) { if (run - own[1] > u) atomicMin(&sh.found[0], 2 * tid); atomicMax(&sh.found[1], 2 * tid); }
    if (own[1] > 0.0) { if (run > u) atomicMin(&sh.found[0], 2 * tid + 1); atomicMax(&sh.found[1], 2 * tid + 1); }
    __syncthreads();
    token = (int) (0xffffffffu - (unsigned) (sh.sorted[sh.found[0] < kListMax ? sh.found[0] : sh.found[1]] >> 32));   // else (rounding) the last
    return true;
}

// The smallest key in front of bin b.  A whole warp calls it: seven rounds of 32 borders.
template <bool STAGED>
__device__ __forceinline__ unsigned bin_border(const Draw<STAGED> & d, int b) {
    unsigned lo = order_key(-INFINITY), hi = draw_key(d.zmax) + 1u;          // in a later bin, and as if in front of the first
    while (hi - lo > 1u) {
        const unsigned long long span = hi - lo;
        const unsigned border = lo + (unsigned) (span * (unsigned) ((threadIdx.x & 31) + 1) >> 5);       // the last lane's is hi
        const bool before = border == hi || (d.zmax - key_value(border)) * kBinsPerUnit < (float) b;
        const int first = __ffs(__ballot_sync(0xffffffffu, before)) - 1;     // borders rise, so that all from here on are
        hi = lo + (unsigned) (span * (unsigned) (first + 1) >> 5);
        lo += (unsigned) (span * (unsigned) first >> 5);
    }
    return hi;
}

// The cut of top-k (0: none) and top-p (>= 1: none) among the keys at or above `cut`, by bins and a sorted list.  1: candidates are the keys
// above the new cut and the first n_tie entries equal to it.  0: not found this way.  2: more entries share the cut's bin than are listed;
// what is known of the bin is in shared memory.  With 0 and 2 cut and n_tie are as before.
template <bool STAGED>
__device__ __forceinline__ int cut_by_bins(const Draw<STAGED> & d, int begin, int V, int k, float P, unsigned & cut, int & n_tie) {
    DrawShared & sh = d.sh;
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool by_k = k > 0;                     // then only counts: the list's own masses are enough for top-p
    // the bins reach as far as the cut may lie: beyond log(V / (1 - P)) all entries together weigh less than 1 - P of the largest one
    const int open = by_k ? kBins - 1 : (int) fminf((logf((float) V) - logf(1.0f - P) + 0.5f) * kBinsPerUnit, (float) (kBins - 1));
    sh.bins.count[tid] = 0;
    sh.bins.low[tid] = sh.bins.high[tid] = 0u;
    if (tid == 0) sh.found[0] = kBins;
    __syncthreads();
    int open_c = 0;                              // the open bin is kept in registers: most of a peaked row falls into it
    unsigned long long open_m = 0ull;
    for (int i0 = tid; i0 < d.n; i0 += 4 * kDrawThreads) {   // four entries side by side: their bins before the first is counted
        int bin[4];
        unsigned q[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u * kDrawThreads;
            const unsigned key = i < d.n ? d.key(i) : 0u;
            const float z = key_value(max(key, cut));
            bin[u] = (int) fminf((d.zmax - z) * kBinsPerUnit, (float) open);
            if (!by_k) q[u] = (unsigned) (expf(z - d.zmax) * __int_as_float((127 + bin_bits(bin[u])) << 23));
            if (key < cut) bin[u] = -1;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (bin[u] == open) {
                open_c++;
                if (!by_k) open_m += q[u];
            } else if (bin[u] >= 0) {
                if (by_k) atomicAdd(&sh.bins.count[bin[u]], 1);
                else { atomicAdd(&sh.bins.low[bin[u]], q[u] & 8191u); atomicAdd(&sh.bins.high[bin[u]], q[u] >> 13); }
            }
        }
    }
    if (open_c > 0) {
        atomicAdd(&sh.bins.count[open], open_c);
        atomicAdd(&sh.bins.low[open], (unsigned) (open_m & 8191u));
        atomicAdd(&sh.bins.high[open], (unsigned) (open_m >> 13));
    }
    cl.sync();                                   // what the CTAs listed before, if they did, has been read too
    if (tid == 0) sh.n_list = 0;
    int c = 0;
    unsigned long long low = 0ull, high = 0ull;
#pragma unroll
    for (int r = 0; r < kDrawCluster; r++) {
        if (r >= d.ctas) break;
        const DrawShared * from = cl.map_shared_rank(&sh, r);
        if (by_k) c += from->bins.count[tid];
        else { low += from->bins.low[tid]; high += from->bins.high[tid]; }
    }
    double m = (double) (low + (high << 13)) * __longlong_as_double((long long) (1023 - bin_bits(tid)) << 52), mass;
    const int own_c = c;
    int count;
    block_scan(sh, c, m, count, mass);           // from the largest values down to this bin
    const double target = (double) P * mass;
    if (by_k ? c >= k && c - own_c < k : m >= target) atomicMin(&sh.found[0], tid);
    __syncthreads();
    const int last = sh.found[0];                // the bin that holds the cut (with both: the one of top-k)
    if (last >= open) return 0;                  // top-k of no effect, or a cut in the open bin
    if (tid == last - 1) { sh.m_above = m; sh.c_above = c; }
    if (tid == last) { sh.m_at = m; sh.c_at = c; sh.target = target; }
    __syncthreads();
    const int first = by_k ? 0 : last;           // with top-k the list begins at the top
    const double m_above = by_k || last == 0 ? 0.0 : sh.m_above;
    // entries to list: counted, or of a bin's mass at the most that one of its entries weighs (up to 4 percent too few)
    if (by_k ? sh.c_at > kListMax : (sh.m_at - m_above) * (double) exp2f((float) last * 0.0625f) > (double) kListMax) return 2;
    for (int i0 = tid; i0 < d.n; i0 += 4 * kDrawThreads) {
        unsigned key[4];
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u * kDrawThreads;
            key[u] = i < d.n ? d.key(i) : 0u;
            const float place = (d.zmax - key_value(max(key[u], cut))) * kBinsPerUnit;
            in[u] = key[u] >= cut && place >= (float) first && place < (float) (last + 1);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (in[u]) {
                const int at = atomicAdd(&sh.n_list, 1);
                if (at < kListMax) sh.list[at] = ((unsigned long long) key[u] << 32) | (0xffffffffu - (unsigned) (begin + i0 + u * kDrawThreads));
            }
    }
    const int n = merge_lists(d);
    if (n > kListMax) return 2;
    if (by_k) {
        block_sort(sh, n);
        const int kept = P < 1.0f ? shortest_run(d, k, P) : k;
        const unsigned at_cut = (unsigned) (sh.sorted[kept - 1] >> 32);
        cut = at_cut;
        __syncthreads();                         // found[1] has been read
        for (int i = tid; i < n; i += kDrawThreads) {
            if ((unsigned) (sh.sorted[i] >> 32) != at_cut) continue;
            if (i == 0 || (unsigned) (sh.sorted[i - 1] >> 32) != at_cut) sh.found[0] = i;
            if (i == n - 1 || (unsigned) (sh.sorted[i + 1] >> 32) != at_cut) sh.found[1] = i;
        }
        __syncthreads();
        n_tie = kept == sh.found[1] + 1 ? 0x7fffffff : kept - sh.found[0];       // all of them, or the first few
        return 1;
    }
    // The largest key whose list entries from there on weigh what is still to reach, in the bin's own whole multiples: every warp weighs
    // one border a pass, and an interval of keys shrinks to a sixteenth.
    const float unit = __int_as_float((127 + bin_bits(last)) << 23);
    const unsigned long long need = (unsigned long long) fmax(ceil((target - m_above) * (double) unit), 1.0);
    if (tid == 0) { sh.lo_key = 0xffffffffu; sh.hi_key = 0u; }
    __syncthreads();
    for (int i = tid; i < n; i += kDrawThreads) {            // (key, ~id) -> (key, weight)
        const unsigned key = (unsigned) (sh.sorted[i] >> 32);
        sh.sorted[i] = ((unsigned long long) key << 32) | (unsigned) (d.mass(key) * unit);
        atomicMin(&sh.lo_key, key);
        atomicMax(&sh.hi_key, key);
    }
    __syncthreads();
    unsigned lo = sh.lo_key, hi = sh.hi_key + 1u;
    unsigned long long q_hi = 0ull;              // what the keys from hi on weigh: less than `need`; from lo on all do (or rounding has it so)
    while (hi - lo > 1u) {
        const unsigned long long span = hi - lo;
        const unsigned border = lo + (unsigned) ((span * (unsigned) (warp + 1)) >> 4);   // the last warp's is hi
        unsigned part = 0u;                      // at most 32 weights of 2^25 a lane
        for (int i = lane; i < n; i += 32) {
            const unsigned long long x = sh.sorted[i];
            part += (unsigned) (x >> 32) >= border ? (unsigned) x : 0u;
        }
        const unsigned q_low = __reduce_add_sync(0xffffffffu, part & 0xffffu), q_high = __reduce_add_sync(0xffffffffu, part >> 16);
        if (lane == 0) sh.warp_q[warp] = ((unsigned long long) q_high << 16) + q_low;
        __syncthreads();
        const unsigned ok = __ballot_sync(0xffffffffu, lane < kDrawWarps - 1 && sh.warp_q[lane & (kDrawWarps - 1)] >= need);
        const int reached = __popc(ok);          // the borders rise: the first of them reach
        if (reached < kDrawWarps - 1) { q_hi = sh.warp_q[reached]; hi = lo + (unsigned) ((span * (unsigned) (reached + 1)) >> 4); }
        lo += (unsigned) ((span * (unsigned) reached) >> 4);
        __syncthreads();
    }
    int ties = 0;
    for (int i = lane; i < n; i += 32) ties += (unsigned) (sh.sorted[i] >> 32) == lo;
    ties = __reduce_add_sync(0xffffffffu, ties);
    const unsigned long long each = (unsigned long long) (d.mass(lo) * unit);
    const unsigned long long some = each > 0ull && need > q_hi ? (need - q_hi + each - 1ull) / each : 1ull;
    cut = lo;
    n_tie = some >= (unsigned long long) ties ? 0x7fffffff : (int) some;         // all of them, or the first few
    return 1;
}

// What bins and lists have not found: an interval of keys is narrowed, all from `cut` to `top` or (near) those of the cut's bin alone, some 2^16 and
// half the passes.  Rows of 151,936, T = 1.0, top-p 0.95 (1,258 entries in the bin): 48 rows 115 us, one 52; from all keys 190 and 80.
// Out of line: the common rows' path loses 10 percent where the compiler has to find registers for this one, too.
struct Cut { unsigned key; int n_tie, turn; };
template <bool STAGED>
__device__ __noinline__ Cut cut_by_passes(Draw<STAGED> d, int begin, int V, int k, float P, unsigned top, unsigned cut, int n_tie, bool near) {
    const int lane = threadIdx.x & 31;
    if (k > 0) {
        unsigned lo = cut, hi = top;
        int count, above = 0;
        if (near) {
            const int bin = d.sh.found[0];
            lo = max(cut, bin_border(d, bin + 1));
            hi = bin_border(d, bin);
            count = d.sh.c_at;
            above = bin > 0 ? d.sh.c_above : 0;
        }
        else {
            int c;
            double m;
            d.template pass<false>(cut, cut, top, c, m);
            count = __shfl_sync(0xffffffffu, c, 0);
        }
        double none = 0.0;
        if (near || k < count) {
            d.template search<false>(lo, hi, count, above, none, (double) k, !near);
            cut = lo;
            n_tie = k - above;
        }
        const bool whole = near && count - above == n_tie;   // no entry equal to the cut was left out: bins serve for top-p
        near = false;
        if (whole && P < 1.0f) {
            cg::this_cluster().sync();           // the bins of this CTA have been read
            const int how = cut_by_bins(d, begin, V, 0, P, cut, n_tie);
            if (how == 1) return {cut, n_tie, d.turn};
            near = how == 2;
        }
    }
    if (P < 1.0f) {
        // the cut moves up to the largest key whose mass from there on reaches the target
        auto move_up = [&](unsigned K, unsigned hi, int c_gt, int c_above, double m_above, double target, bool wide) {
            d.template search<true>(K, hi, c_gt, c_above, m_above, target, wide);
            const int tie_p = c_gt - c_above;
            const float pe = d.mass(K);
            const int need = pe > 0.0f ? (int) fmin(ceil((target - m_above) / (double) pe), 2147483647.0) : tie_p;
            cut = K;
            n_tie = max(1, min(need, tie_p));
        };
        if (near) {                              // (of the counts only those of a pass are needed)
            const int bin = d.sh.found[0];
            move_up(max(cut, bin_border(d, bin + 1)), bin_border(d, bin), 0x7fffffff, 0, bin > 0 ? d.sh.m_above : 0.0, d.sh.target, false);
        } else {
            // borders: cut in lane 0, cut + 1 in the others (entries equal to the cut: the difference of the counts)
            int c;
            double m;
            d.template pass<true>(cut + (lane > 0 ? 1u : 0u), cut, top, c, m);
            const int c_all = __shfl_sync(0xffffffffu, c, 0), c_gt = __shfl_sync(0xffffffffu, c, 1);
            const double m_gt = __shfl_sync(0xffffffffu, m, 1);
            const int ties_in = min(c_all - c_gt, n_tie);
            const float pe_cut = ties_in > 0 ? d.mass(cut) : 0.0f;
            const double target = (double) P * (m_gt + (double) ties_in * (double) pe_cut);
            if (target > 0.0 && m_gt >= target) move_up(cut + 1, top, c_gt, 0, 0.0, target, true);
            else if (ties_in > 0 && pe_cut > 0.0f) {
                const int need = (int) fmin(ceil((target - m_gt) / (double) pe_cut), 2147483647.0);
                n_tie = max(m_gt >= target ? 0 : 1, min(need, ties_in));
                if (m_gt <= 0.0) n_tie = max(n_tie, 1);
            }
        }
    }
    return {cut, n_tie, d.turn};
}

// A row's settings: from arrays on the device, or from the launch's own parameters (no copy in front of it).
struct SettingArrays {
    const float * temperature_, * top_p_, * min_p_, * uniform_;
    const int * top_k_;
    __device__ __forceinline__ float temperature(int r) const { return temperature_[r]; }
    __device__ __forceinline__ float top_p(int r) const { return top_p_[r]; }
    __device__ __forceinline__ float min_p(int r) const { return min_p_[r]; }
    __device__ __forceinline__ float uniform(int r) const { return uniform_[r]; }
    __device__ __forceinline__ int top_k(int r) const { return top_k_[r]; }
};
constexpr int kRowsAtOnce = 128;                 // rows of a launch whose settings are parameters: 2.5 of 4 KB
struct SettingRows {
    float temperature_[kRowsAtOnce], top_p_[kRowsAtOnce], min_p_[kRowsAtOnce], uniform_[kRowsAtOnce];
    int top_k_[kRowsAtOnce];
    __device__ __forceinline__ float temperature(int r) const { return temperature_[r]; }
    __device__ __forceinline__ float top_p(int r) const { return top_p_[r]; }
    __device__ __forceinline__ float min_p(int r) const { return min_p_[r]; }
    __device__ __forceinline__ float uniform(int r) const { return uniform_[r]; }
    __device__ __forceinline__ int top_k(int r) const { return top_k_[r]; }
};

template <bool STAGED, typename Settings>
__global__ void __launch_bounds__(kDrawThreads, 2) sample_kernel(
    const float * __restrict__ logits, int V, size_t stride, int slice, const __grid_constant__ Settings set, int * __restrict__ out) {
    extern __shared__ unsigned staged[];
    __shared__ DrawShared sh;
    __shared__ float fs[32];
    __shared__ int is[32];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ctas = (int) cl.num_blocks(), rank = (int) cl.block_rank(), row = blockIdx.x / ctas;
    const int begin = (int) min((long long) V, (long long) rank * slice), n = (int) min((long long) V, (long long) begin + slice) - begin;
    const float * src = logits + (size_t) row * stride + begin;
    const float T = set.temperature(row);
    const bool greedy = T < 1e-5f;
    const float inv_t = greedy ? 1.0f : 1.0f / T;

    // the slice into shared memory; the row's largest value and the lowest id that holds it
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    auto take = [&](int i, float v) {
        const float z = v * inv_t;
        if (STAGED) staged[i] = draw_key(z);
        if (z > best || (z == best && begin + i < best_i)) { best = z; best_i = begin + i; }        // NaN compares false
    };
    for (int base = 0; base < n; base += kAsked * kDrawThreads) {
        const int rounds = min((n - base) / kDrawThreads, kAsked), at = base + tid, last = at + rounds * kDrawThreads;
        const bool more = rounds < kAsked && last < n;       // the round that not all threads have an entry of
        float v[kAsked], w = 0.0f;
#pragma unroll
        for (int u = 0; u < kAsked; u++) {
            if (u >= rounds) break;
            v[u] = src[at + u * kDrawThreads];
        }
        if (more) w = src[last];
#pragma unroll
        for (int u = 0; u < kAsked; u++) {
            if (u >= rounds) break;
            take(at + u * kDrawThreads, v[u]);
        }
        if (more) take(last, w);
    }
    auto better = [&](float ob, int oi) { if (ob > best || (ob == best && oi < best_i)) { best = ob; best_i = oi; } };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        better(ob, oi);
    }
    if (lane == 0) { fs[warp] = best; is[warp] = best_i; }
    cl.sync();                                   // every CTA of the cluster runs before its shared memory is written; orders fs, is and staged too
    Draw<STAGED> d{sh, staged, src, n, inv_t, 0.0f, rank, ctas, 0};
    if (warp == 0) {
        best = lane < kDrawWarps ? fs[lane] : -INFINITY;
        best_i = lane < kDrawWarps ? is[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            better(ob, oi);
        }
        if (STAGED && lane < kDrawWarps)         // the warps' largest values too
            for (int r = 0; r < ctas; r++) cl.map_shared_rank(&sh, r)->tops[rank * kDrawWarps + lane] = fs[lane];
        d.send(lane, 0, (double) best, best_i);
    }
    d.swap();
    best = -INFINITY;
    best_i = 0x7fffffff;
    for (int r = 0; r < ctas; r++) better((float) sh.inbox_m[d.turn][r][0], sh.inbox_c[d.turn][r][0]);
    d.turn ^= 1;
    const int imax = best_i == 0x7fffffff ? 0 : best_i;
    d.zmax = best;
    const float P = set.top_p(row);
    // nothing to draw from: a greedy row, an infinite or missing largest value, or a share of the mass that keeps none (these
    // tests see the same numbers in every CTA, so a cluster leaves together; what was sent has been read by its receiver only
    // after the barrier above, and nothing is sent after it)
    if (greedy || !(fabsf(best) < INFINITY) || P <= 0.0f) {
        if (rank == 0 && tid == 0) out[row] = imax;
        return;
    }
    const unsigned top = draw_key(best) + 1;     // above every key
    // candidates: keys above `cut`, and the first n_tie entries (by id) whose key is `cut`
    unsigned cut = order_key(-INFINITY) + 1u;    // entries without mass change nothing
    int n_tie = 0x7fffffff;
    const float mp = set.min_p(row);
    if (mp > 0.0f) cut = max(cut, order_key(best + logf(mp)));
    const int k = set.top_k(row);
    const bool cuts = cut < top && (k > 0 || P < 1.0f);
    if (STAGED && cuts && k > 0 && k <= ctas * kDrawWarps / 2) {
        int token;
        if (draw_from_list(d, begin, k, P, cut, set.uniform(row), token)) {
            if (rank == 0 && tid == 0) out[row] = token;
            cl.sync();                           // the lists of this CTA have been read
            return;
        }
    }
    const int how = STAGED && cuts ? cut_by_bins(d, begin, V, k, P, cut, n_tie) : 0;
    if (cuts && how != 1) {
        const Cut now = cut_by_passes(d, begin, V, k, P, top, cut, n_tie, how == 2);
        cut = now.key;
        n_tie = now.n_tie;
        d.turn = now.turn;
    }

    // inverse CDF in vocabulary order: thread t owns `per` neighbouring entries (an odd number: no two lanes in one bank)
    const int per = ((n + kDrawThreads - 1) / kDrawThreads) | 1;
    const int i0 = (int) min((long long) n, (long long) tid * per), i1 = min(n, i0 + per);
    int ties = 0, tie_rank = 0;
    if (n_tie != 0x7fffffff) {                   // else every entry equal to the cut stays
        for (int i = i0; i < i1; i++) ties += d.key(i) == cut;
        tie_rank = ties;                         // inclusive scan over the CTA, then the CTAs before
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, tie_rank, o);
            if (lane >= o) tie_rank += v;
        }
        __syncthreads();                             // sh.warp_i may still be read from the search
        if (lane == 31) sh.warp_i[warp] = tie_rank;
        __syncthreads();
        if (warp == 0) {
            const int w = lane < kDrawWarps ? sh.warp_i[lane] : 0;
            d.send(lane, 0, 0.0, __reduce_add_sync(0xffffffffu, w));
        }
        d.swap();
        tie_rank -= ties;
        for (int w = 0; w < warp; w++) tie_rank += sh.warp_i[w];
        for (int r = 0; r < rank; r++) tie_rank += sh.inbox_c[d.turn][r][0];
        d.turn ^= 1;
    }
    double cm = 0.0;
    int tr = tie_rank;
#pragma unroll 4
    for (int i = i0; i < i1; i++) {
        const unsigned kk = d.key(i);
        if (kk > cut) cm += (double) d.mass(kk);
        else if (kk == cut) { if (tr < n_tie) cm += (double) d.mass(kk); tr++; }
    }
    double incl = cm;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) sh.warp_d[warp] = incl;
    if (tid == 0) sh.pick = -1;
    __syncthreads();
    double before = 0.0, all = 0.0;
    for (int w = 0; w < kDrawWarps; w++) {
        if (w == warp) before = all;
        all += sh.warp_d[w];
    }
    if (warp == 0) d.send(lane, 0, all, 0);
    d.swap();
    double total = 0.0;
    for (int r = 0; r < ctas; r++) total += sh.inbox_m[d.turn][r][0];
    const double u = (double) set.uniform(row) * total;
    // the CTA the draw falls into: the first whose running sum passes it, else (rounding) the last that holds mass
    int owner = -1;
    double run = 0.0, ahead = 0.0;
    for (int r = 0; r < ctas; r++) {
        const double v = sh.inbox_m[d.turn][r][0];
        if (v > 0.0) { owner = r; ahead = run; if (run + v > u) break; }
        run += v;
    }
    if (owner < 0) {                             // no candidate holds mass
        if (rank == 0 && tid == 0) out[row] = imax;
        return;
    }
    if (rank != owner) return;
    // the thread: the same way
    const double lead = ahead + before;
    if (cm > 0.0) atomicMax(&sh.pick, lead + incl > u ? kDrawThreads * 2 - tid : tid);     // the first past the draw, else the last
    __syncthreads();
    const int pick = sh.pick >= kDrawThreads ? kDrawThreads * 2 - sh.pick : sh.pick;
    if (tid != pick) return;
    double at = lead + (incl - cm);
    int chosen = -1, last = -1;
    tr = tie_rank;
    for (int i = i0; i < i1; i++) {
        const unsigned kk = d.key(i);
        float e = 0.0f;
        if (kk > cut) e = d.mass(kk);
        else if (kk == cut) { if (tr < n_tie) e = d.mass(kk); tr++; }
        if (e > 0.0f) {
            last = i;
            at += (double) e;
            if (at > u) { chosen = i; break; }
        }
    }
    if (chosen < 0) chosen = last;
    out[row] = chosen >= 0 ? begin + chosen : imax;
}

// Logits processors in the reference's order (src/iian/sampler.cpp:72-109), as lists the host prepares per row:
//  * allowed ids (sorted; an empty list allows everything): every other logit becomes -inf (:72-76);
//  * one edit per touched token: l += pre (logit bias; -inf for a banned token or the end of a bad word, :77-88),
//    then l = l > 0 ? l * mul_pos : l * mul_neg (repetition penalty: 1 / r and r, :106), then l += post
//    (-(frequency * count + presence) for tokens that were produced, :107).
// One block per row; a row's lists are the ranges [off[r], off[r + 1]).
__global__ void logit_edits_kernel(float * __restrict__ logits, int V, size_t stride,
                                   const int * __restrict__ allow_off, const int * __restrict__ allow_ids,
                                   const int * __restrict__ edit_off, const int * __restrict__ edit_tok,
                                   const float * __restrict__ pre, const float * __restrict__ mul_pos,
                                   const float * __restrict__ mul_neg, const float * __restrict__ post) {
    const int r = blockIdx.x;
    float * row = logits + (size_t) r * stride;
    const int a0 = allow_off[r], a1 = allow_off[r + 1];
    if (a1 > a0) {
        for (int v = threadIdx.x; v < V; v += blockDim.x) {
            int lo = a0, hi = a1;                 // is v among the sorted ids [a0, a1)?
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (allow_ids[mid] < v) lo = mid + 1; else hi = mid;
            }
            if (lo == a1 || allow_ids[lo] != v) row[v] = -INFINITY;
        }
        __syncthreads();
    }
    for (int e = edit_off[r] + threadIdx.x; e < edit_off[r + 1]; e += blockDim.x) {
        const int t = edit_tok[e];
        if (t < 0 || t >= V) continue;
        float l = row[t] + pre[e];
        l = l > 0.0f ? l * mul_pos[e] : l * mul_neg[e];
        row[t] = l + post[e];
    }
}

// Log-probabilities of the raw distribution (src/iian/sampler.cpp:63-70, 174-182): log softmax of the row at the
// chosen token and at the k largest logits (value descending, lowest id first among equals).  One block per row;
// the k-th pick is the largest entry that comes after the pick before it in that order, so no entry is marked.
__global__ void __launch_bounds__(kSampleThreads) logprobs_kernel(
    const float * __restrict__ logits, int V, size_t stride, const int * __restrict__ tokens, const int * __restrict__ want_k,
    int kmax, float * __restrict__ out_lp, int * __restrict__ top_ids, float * __restrict__ top_lp) {
    __shared__ float fs[32];
    __shared__ int is[32];
    __shared__ float red[32];
    const int r = blockIdx.x;
    const int k = want_k[r];
    if (k < 0) return;
    const float * row = logits + (size_t) r * stride;
    float mx; int mi;
    block_argmax(row, V, 1.0f, mx, mi, fs, is);
    float acc = 0.0f;
    for (int i = threadIdx.x; i < V; i += blockDim.x) acc += expf(row[i] - mx);
    __syncthreads();
    const float lse = mx + logf(block_sum(acc, red));
    if (threadIdx.x == 0) {
        const int t = tokens[r];
        out_lp[r] = (t >= 0 && t < V) ? row[t] - lse : -INFINITY;
    }
    float pv = INFINITY;
    int pi = -1;
    for (int j = 0; j < kmax; j++) {
        if (j >= k || j >= V) {
            if (threadIdx.x == 0) { top_ids[(size_t) r * kmax + j] = -1; top_lp[(size_t) r * kmax + j] = -INFINITY; }
            continue;
        }
        float b = -INFINITY;
        int bi = 0x7fffffff;
        for (int i = threadIdx.x; i < V; i += blockDim.x) {
            const float v = row[i];
            const bool after = v < pv || (v == pv && i > pi);          // after the pick before, in (value desc, id asc) order
            if (after && (v > b || (v == b && i < bi))) { b = v; bi = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, b, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        __syncthreads();
        if (lane == 0) { fs[warp] = b; is[warp] = bi; }
        __syncthreads();
        b = lane < (blockDim.x >> 5) ? fs[lane] : -INFINITY;
        bi = lane < (blockDim.x >> 5) ? is[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, b, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > b || (ob == b && oi < bi)) { b = ob; bi = oi; }
        }
        pv = b; pi = bi;
        if (threadIdx.x == 0) {
            top_ids[(size_t) r * kmax + j] = bi == 0x7fffffff ? -1 : bi;
            top_lp[(size_t) r * kmax + j] = bi == 0x7fffffff ? -INFINITY : b - lse;
        }
    }
}

}  // namespace iian

using namespace iian;

IIAN_API int iian_argmax(const float * logits, int R, int V, long long stride, int * out, cudaStream_t stream) {
    if (R <= 0) return IIAN_OK;
    if (V <= 0) return IIAN_ERR_SHAPE;
    argmax_kernel<<<R, kSampleThreads, 0, stream>>>(logits, V, (size_t) stride, out);
    return iian_launch_status();
}

// Wide rows: scratch must hold R * parts floats followed by R * parts ints (parts = iian_argmax_parts(V)).
IIAN_API int iian_argmax_parts(int V) { return V >= 16384 ? 64 : 0; }

IIAN_API int iian_argmax_wide(const float * logits, int R, int V, long long stride, void * scratch, int * out,
                              cudaStream_t stream) {
    if (R <= 0) return IIAN_OK;
    const int parts = iian_argmax_parts(V);
    if (V <= 0 || parts == 0 || scratch == nullptr || R > 65535) return IIAN_ERR_SHAPE;
    float * pv = (float *) scratch;
    int * pi = (int *) (pv + (size_t) R * parts);
    const int rc = iian_launch(argmax_partial_kernel, dim3(parts, R), dim3(256), 0, stream, logits, V, (size_t) stride, parts, pv, pi);
    if (rc != IIAN_OK) return rc;
    return iian_launch(argmax_final_kernel, dim3(R), dim3(32), 0, stream, (const float *) pv, (const int *) pi, parts, out);
}

// CTAs per row: slices of up to 13,000 entries, up to 8 CTAs.  Less of a slice is no faster for a few rows and a wave more for many: 48 rows
// of 32,768 with 8 CTAs 31 us, with 4 22, with 2 27; of 50,257 with 8 35, with 4 29; 16 CTAs of a row of 151,936 72 for 49 with 8.
template <typename Settings>
static int launch_sample(const float * logits, int R, int V, long long stride, const Settings & set, int * out, cudaStream_t stream) {
    int ctas = 1;
    while (ctas < kDrawCluster && V > ctas * kSliceGoal) ctas *= 2;
    const int slice = (V - 1) / ctas + 1;
    const bool staged = slice <= kStagedMax;
    const size_t smem = staged ? (size_t) slice * sizeof(unsigned) : 0;
    auto kernel = staged ? sample_kernel<true, Settings> : sample_kernel<false, Settings>;
    if (smem > 24 * 1024) {                      // with the 20 KB of static memory above what a launch may ask for by itself
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        if (e != cudaSuccess) return 1000 + (int) e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kDrawThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned) ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned) R * (unsigned) ctas);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, logits, V, (size_t) stride, slice, set, out);
    return e == cudaSuccess ? IIAN_OK : 1000 + (int) e;
}

IIAN_API int iian_sample(const float * logits, int R, int V, long long stride, const float * temperature,
                         const int * top_k, const float * top_p, const float * min_p, const float * uniform,
                         int * out, cudaStream_t stream) {
    if (R <= 0) return IIAN_OK;
    if (V <= 0) return IIAN_ERR_SHAPE;
    return launch_sample(logits, R, V, stride, SettingArrays{temperature, top_p, min_p, uniform, top_k}, out, stream);
}

static inline unsigned long long splitmix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// The same with the rows' settings on the host: (temperature, top_p, min_p) a row, top_k, and number `index` of the row's stream of uniform
// numbers, a hash of (seed, index).  They travel as launch parameters, kRowsAtOnce rows a launch.  out may be pinned host memory: it
// holds the tokens once the stream has been waited for.
IIAN_API int iian_sample_rows(const float * logits, int R, int V, long long stride, const float * settings, const int * top_k,
                              const unsigned long long * seeds, const unsigned long long * indices, int * out, cudaStream_t stream) {
    if (R <= 0) return IIAN_OK;
    if (V <= 0 || settings == nullptr || top_k == nullptr || seeds == nullptr || indices == nullptr) return IIAN_ERR_SHAPE;
    for (int r0 = 0; r0 < R; r0 += kRowsAtOnce) {
        const int n = R - r0 < kRowsAtOnce ? R - r0 : kRowsAtOnce;
        SettingRows set;
        for (int r = 0; r < n; r++) {
            set.temperature_[r] = settings[3 * (r0 + r)];
            set.top_p_[r] = settings[3 * (r0 + r) + 1];
            set.min_p_[r] = settings[3 * (r0 + r) + 2];
            set.top_k_[r] = top_k[r0 + r];
            const unsigned long long h = splitmix64(splitmix64(seeds[r0 + r]) ^ (indices[r0 + r] * 0xD1B54A32D192ED03ull));
            set.uniform_[r] = (float) (h >> 40) * 5.9604644775390625e-8f;                      // 2^-24: 24 bits, exact
        }
        const int rc = launch_sample(logits + (size_t) r0 * stride, n, V, stride, set, out + r0, stream);
        if (rc != IIAN_OK) return rc;
    }
    return IIAN_OK;
}

// logits [R, V] float32, changed in place.  allow_off / edit_off: [R + 1] int32 prefix sums; a token may appear in
// at most one edit of its row.
IIAN_API int iian_logit_edits(float * logits, int R, int V, long long stride, const int * allow_off, const int * allow_ids,
                              const int * edit_off, const int * edit_tok, const float * pre, const float * mul_pos,
                              const float * mul_neg, const float * post, cudaStream_t stream) {
    if (R <= 0) return IIAN_OK;
    if (V <= 0 || allow_off == nullptr || edit_off == nullptr) return IIAN_ERR_SHAPE;
    logit_edits_kernel<<<R, 256, 0, stream>>>(logits, V, (size_t) stride, allow_off, allow_ids, edit_off, edit_tok, pre,
                                              mul_pos, mul_neg, post);
    return iian_launch_status();
}

// Raw log-probabilities: out_lp [R] at tokens [R]; the want_k[r] (at most kmax; negative: skip the row) largest
// entries of row r into top_ids / top_lp [R, kmax], the rest of a row filled with -1 / -inf.
IIAN_API int iian_logprobs(const float * logits, int R, int V, long long stride, const int * tokens, const int * want_k,
                           int kmax, float * out_lp, int * top_ids, float * top_lp, cudaStream_t stream) {
    if (R <= 0) return IIAN_OK;
    if (V <= 0 || kmax < 0 || kmax > 64) return IIAN_ERR_SHAPE;
    logprobs_kernel<<<R, kSampleThreads, 0, stream>>>(logits, V, (size_t) stride, tokens, want_k, kmax, out_lp, top_ids, top_lp);
    return iian_launch_status();
}
