// Paged attention, general form: any element type, head size, number of heads and groups, page
// size and window.  One warp per (token, head); keys are walked in tiles of 32 that start at
// multiples of 32 of the ABSOLUTE key position, so the order of every sum depends only on the
// token's own position -- not on how the request was cut into steps or what else is in the batch.
// This is the whole attention of the 32-bit path and the fallback of the bfloat16 path for sizes
// the tensor-core kernels do not take.
//
// Formula (reference): head h reads KV head h / (nh / nkv); s_j = (q . k_j) * scale; key j is
// visible iff j <= pos and (window == 0 or pos - j < window); softmax in float32; o = sum p_j v_j
// (src/iian/paged_attn.cpp:112-145, window test :124).
//
// Two options beyond the reference's formula, for mixers that have them: a sink per head (a logit with no key and no
// value that joins the softmax's denominator once, unscaled: the running softmax simply starts at maximum sink_h with
// denominator 1), and an output gate (o *= sigmoid(g) element by element, g read from rows of a wider matrix).
#include <type_traits>

#include "common.cuh"
#include "packed.cuh"

namespace iian {

constexpr int kGenMaxHeadDim = 512;
constexpr int kGenWarps = 4;

constexpr int kTileItems = 32;      // (token, head) pairs of a CTA of the tiled kernel: 32 / (heads of a group) tokens
constexpr int kTileRuns = 4;        // requests whose tokens may lie side by side in such a CTA
constexpr int kTileMinTokens = 8;   // tokens of a step from which the tiled kernel is launched

// Whether the tokens [t0, t0 + tokens) of the step are the tiled kernel's: at most kTileRuns runs of a request's tokens, two tokens each on
// average (a CTA walks the runs one after the other: decoded tokens are better off with a warp for every item side by side) unless they
// are the end of a longer portion, and no padding.  Both kernels ask.  A whole warp calls it (at most 32 tokens a tile).
__device__ __forceinline__ bool tile_is_shared(const int * __restrict__ seq_of_token, int t0, int tokens, int N) {
    const int lane = threadIdx.x & 31;
    const bool in = lane < tokens && t0 + lane < N;
    const int s = in ? seq_of_token[t0 + lane] : 0;
    const int before = __shfl_up_sync(0xffffffffu, s, 1);
    const unsigned padding = __ballot_sync(0xffffffffu, in && s < 0), starts = __ballot_sync(0xffffffffu, in && (lane == 0 || s != before));
    const int runs = __popc(starts), n = min(tokens, N - t0);
    const int ahead = t0 > 0 ? seq_of_token[t0 - 1] : -1, first = __shfl_sync(0xffffffffu, s, 0);
    return padding == 0 && runs <= kTileRuns && (n >= 2 * runs || (runs == 1 && ahead == first));
}

// VEC: rows of keys are whole 16-byte pieces.  NACC: output entries per lane (hd <= 32 * NACC).
template <typename A, int NACC, bool VEC>
__global__ void paged_attention_generic_kernel(
    const A * __restrict__ q, const A * __restrict__ k_cache, const A * __restrict__ v_cache,
    A * __restrict__ out, const int * __restrict__ positions, const int * __restrict__ seq_of_token,
    const int * __restrict__ block_table, int max_blocks, const int * __restrict__ ctx_len,
    int N, int nh, int nkv, int hd, int page_size, int num_pages, float scale, int window,
    const float * __restrict__ sink, const A * __restrict__ gate, long long ld_gate, int tile_tokens) {
    __shared__ __align__(16) float qs[kGenWarps][kGenMaxHeadDim];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long) blockIdx.x * kGenWarps + warp;
    if (item >= (long long) N * nh) return;
    const int t = (int) (item / nh), h = (int) (item % nh);
    if (tile_tokens > 0 && tile_is_shared(seq_of_token, t / tile_tokens * tile_tokens, tile_tokens, N)) return;
    const int kvh = h / (nh / nkv);
    A * o = out + ((size_t) t * nh + h) * hd;
    const int s = seq_of_token[t];
    if (s < 0) {   // padding token
        for (int d = lane; d < hd; d += 32) o[d] = from_f32<A>(0.0f);
        return;
    }
    const int p = positions[t];
    int hi = p;
    if (ctx_len != nullptr) hi = min(hi, ctx_len[s] - 1);
    const int lo = window > 0 ? max(0, p - window + 1) : 0;

    const A * qp = q + ((size_t) t * nh + h) * hd;
    for (int d = lane; d < hd; d += 32) qs[warp][d] = to_f32(qp[d]);
    __syncwarp();

    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; i++) acc[i] = 0.0f;
    float m = sink != nullptr ? sink[h] : -INFINITY, l = sink != nullptr ? 1.0f : 0.0f;
    const int * bt = block_table + (size_t) s * max_blocks;

    for (int kb = (lo / 32) * 32; kb <= hi; kb += 32) {
        const int j = kb + lane;
        bool valid = j >= lo && j <= hi;
        const A * kp = nullptr;
        const A * vp = nullptr;
        if (valid) {
            const int page = bt[j / page_size];
            if (page < 0 || page >= num_pages) {
                valid = false;      // a page that was given back is never inside the window; never read it
            } else {
                const size_t cell = (((size_t) page * nkv + kvh) * page_size + (j % page_size)) * hd;
                kp = k_cache + cell;
                vp = v_cache + cell;
            }
        }
        float sc = -INFINITY;
        if (valid) {
            float dot = 0.0f;
            if (VEC) {
                constexpr int PIECE = 16 / sizeof(A);
#pragma unroll 8
                for (int d = 0; d < hd; d += PIECE) {
                    const uint4 raw = __ldg(reinterpret_cast<const uint4 *>(kp + d));
                    const A * kk = reinterpret_cast<const A *>(&raw);
#pragma unroll
                    for (int e = 0; e < PIECE; e++) dot = fmaf(qs[warp][d + e], to_f32(kk[e]), dot);
                }
            } else
                for (int d = 0; d < hd; d++) dot = fmaf(qs[warp][d], to_f32(kp[d]), dot);
            sc = dot * scale;
        }
        const float tile_max = warp_max(sc);
        if (tile_max == -INFINITY) continue;
        const float m_new = fmaxf(m, tile_max);
        const float pj = valid ? expf(sc - m_new) : 0.0f;
        const float corr = (m == -INFINITY) ? 0.0f : expf(m - m_new);
        l = l * corr + warp_sum(pj);
#pragma unroll
        for (int i = 0; i < NACC; i++) acc[i] *= corr;
        m = m_new;
        // value rows loaded before the first is added (heads of 160 to 256, 8 bfloat16 tokens behind 1,000: two rows 529 and 696 us, four 921 and
        // 1,333, eight 919 and 1,324; a row at a time over 16 entries a lane 795 and 1,152)
        constexpr int AT_ONCE = NACC <= 4 ? 8 : NACC <= 8 ? 2 : 4;
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += AT_ONCE) {
            float pr[AT_ONCE], vr[AT_ONCE][NACC];
#pragma unroll
            for (int e = 0; e < AT_ONCE; e++) {
                pr[e] = __shfl_sync(0xffffffffu, pj, j0 + e);
                const A * vrow = (const A *) __shfl_sync(0xffffffffu, (unsigned long long) vp, j0 + e);
#pragma unroll
                for (int i = 0; i < NACC; i++) {
                    const int d = lane + 32 * i;
                    vr[e][i] = pr[e] != 0.0f && d < hd ? to_f32(vrow[d]) : 0.0f;
                }
            }
#pragma unroll
            for (int e = 0; e < AT_ONCE; e++) {
                if (pr[e] == 0.0f) continue;
#pragma unroll
                for (int i = 0; i < NACC; i++) acc[i] = fmaf(pr[e], vr[e][i], acc[i]);
            }
        }
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;     // a row that sees no key yields zeros
#pragma unroll
    for (int i = 0; i < NACC; i++) {
        const int d = lane + 32 * i;
        if (d < hd) {
            float v = acc[i] * inv;
            if (gate != nullptr) v *= 1.0f / (1.0f + expf(-to_f32(gate[(size_t) t * ld_gate + h * hd + d])));
            o[d] = from_f32<A>(v);
        }
    }
}

// The same attention in float32 for neighbouring tokens: a CTA owns 32 (token, head) items of one KV head, four a warp, and its key
// tiles -- the same 32 keys from the same multiples of 32 -- come once through two stages of shared memory for all of them.  Every
// item's arithmetic is the kernel's above term by term (a lane is a key in the scores and four output entries in the sum; packed
// multiply-adds of two items, or of two entries, round as single ones do), so an item has the same bits whichever kernel it falls to.
// What bounds it: reads of shared memory.  A warp's 16-byte read of one key row a lane takes 4 clocks, of one address for all lanes 2: a
// tile's scores are 3,072 clocks of an SM, its sums 1,536 (measured 3,100 and about 1,600, copies 1,300, the softmax 1,300 with its
// shuffles for four items side by side).  Eight warps of four items, so that a scheduler has two to choose from, and a page looked up
// a tile before its copy.  2 requests, 301 tokens x 16 heads of 128: 44 us (four warps of eight items, an item's softmax after
// another's: 72; a warp per item, each reading its keys row by row from global memory: 487).
constexpr int kTileHeadDim = 128;
constexpr int kTileWarps = 8, kWarpItems = kTileItems / kTileWarps;
constexpr int kTileLd = kTileHeadDim + 4;
constexpr size_t kTileSmem = (size_t) (2 * 2 * 32 * kTileLd + kTileItems * kTileHeadDim + kTileItems * 32) * sizeof(float);

__global__ void __launch_bounds__(kTileWarps * 32)
paged_attention_tile_kernel(
    const float * __restrict__ q, const float * __restrict__ k_cache, const float * __restrict__ v_cache,
    float * __restrict__ out, const int * __restrict__ positions, const int * __restrict__ seq_of_token,
    const int * __restrict__ block_table, int max_blocks, const int * __restrict__ ctx_len,
    int N, int nh, int nkv, int hd, int page_size, int num_pages, float scale, int window,
    const float * __restrict__ sink, const float * __restrict__ gate, long long ld_gate) {
    extern __shared__ __align__(16) float sm[];
    float * stages = sm;                               // [2][keys | values][32][kTileLd]
    float * qs = sm + 2 * 2 * 32 * kTileLd;            // [16 pairs of items][hd][2]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float * ps = qs + kTileItems * kTileHeadDim + warp * kWarpItems * 32;       // [items of a warp][32 keys]: probabilities
    __shared__ unsigned char good[2][kTileWarps];      // keys of a stage whose page exists, four a warp
    const int G = nh / nkv, tokens = kTileItems / G;
    const int t0 = blockIdx.x * tokens, kvh = blockIdx.y;
    if (!tile_is_shared(seq_of_token, t0, tokens, N)) return;
    const int n_tok = min(tokens, N - t0), n_items = n_tok * G;
    {                                                  // eight threads an item
        const int item = tid >> 3;
        const float * from = q + ((size_t) (t0 + item / G) * nh + kvh * G + item % G) * hd;
        float * to = qs + (item >> 1) * hd * 2 + (item & 1);
        float4 v[kTileHeadDim / 32];
#pragma unroll
        for (int u = 0; u < kTileHeadDim / 32; u++) {
            const int d = ((tid & 7) + 8 * u) * 4;
            v[u] = item < n_items && d < hd ? __ldg(reinterpret_cast<const float4 *>(from + d)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int u = 0; u < kTileHeadDim / 32; u++) {
            const int d = ((tid & 7) + 8 * u) * 4;
            if (d < hd) {
                to[d * 2] = v[u].x; to[d * 2 + 2] = v[u].y;
                to[d * 2 + 4] = v[u].z; to[d * 2 + 6] = v[u].w;
            }
        }
    }
    unsigned long long acc[kWarpItems][2];
    float m[kWarpItems], l[kWarpItems];
    int lo[kWarpItems], hi[kWarpItems], tok[kWarpItems];                          // first and last key; the token, -1: no item
#pragma unroll
    for (int i = 0; i < kWarpItems; i++) {
        const int item = warp * kWarpItems + i, t = t0 + item / G;
        const bool real = item < n_items;
        const float sk = sink != nullptr ? sink[kvh * G + item % G] : -INFINITY;
        m[i] = sk;
        l[i] = sink != nullptr ? 1.0f : 0.0f;
        tok[i] = real ? t : -1;
        const int p = real ? positions[t] : -1;
        hi[i] = real && ctx_len != nullptr ? min(p, ctx_len[seq_of_token[t]] - 1) : p;
        lo[i] = window > 0 ? max(0, p - window + 1) : 0;
        acc[i][0] = acc[i][1] = 0ull;
    }
    const int pieces = hd / 4;
    // a lane per token: its request, last key and first key, so that a run's are found without a walk through memory
    const int my_seq = lane < n_tok ? seq_of_token[t0 + lane] : -1;
    int my_hi = lane < n_tok ? positions[t0 + lane] : -1;
    const int my_lo = lane < n_tok && window > 0 ? max(0, my_hi - window + 1) : 0;
    if (lane < n_tok && ctx_len != nullptr) my_hi = min(my_hi, ctx_len[my_seq] - 1);
    int first = t0;
    while (first < t0 + n_tok) {                       // run after run of one request's tokens; an item walks the keys in its own run alone
        const int begin = first, s = __shfl_sync(0xffffffffu, my_seq, begin - t0);
        const unsigned others = __ballot_sync(0xffffffffu, lane < n_tok && my_seq != s) & (0xffffffffu << (begin - t0));
        const int end = others ? t0 + __ffs(others) - 1 : t0 + n_tok;
        const bool mine = lane >= begin - t0 && lane < end - t0;
        const int k_hi = __reduce_max_sync(0xffffffffu, mine ? my_hi : -1), k_lo = __reduce_min_sync(0xffffffffu, mine ? my_lo : 0x7fffffff);
        first = end;
        int last[kWarpItems];                                   // the items' last keys in this run, -1: the item is another run's
#pragma unroll
        for (int i = 0; i < kWarpItems; i++) last[i] = tok[i] >= begin && tok[i] < end ? hi[i] : -1;
        const int * bt = block_table + (size_t) s * max_blocks;
        const int kb0 = (k_lo / 32) * 32;
        auto page_of = [&](int j) { return j <= k_hi ? bt[j / page_size] : -1; };
        int next_page = page_of(kb0 + (tid >> 3));     // looked up a tile ahead of its copy
        auto fill = [&](int kb, int stage) {           // eight lanes a key
            if (kb <= k_hi) {
                const int r = tid >> 3, j = kb + r, page = next_page;
                next_page = page_of(kb + 32 + r);
                const bool ok = page >= 0 && page < num_pages;
                const size_t cell = ok ? (((size_t) page * nkv + kvh) * page_size + (j % page_size)) * hd : 0;
                float * to = stages + (size_t) stage * 2 * 32 * kTileLd + r * kTileLd;
                for (int c = tid & 7; c < pieces; c += 8) {
                    copy16(to + c * 4, k_cache + cell + c * 4, ok);
                    copy16(to + 32 * kTileLd + c * 4, v_cache + cell + c * 4, ok);
                }
                const unsigned b = __ballot_sync(0xffffffffu, ok);       // this warp's four keys, eight bits each
                if (lane == 0) good[stage][warp] = (unsigned char) ((b & 1u) | (b >> 7 & 2u) | (b >> 14 & 4u) | (b >> 21 & 8u));
            }
            asm volatile("cp.async.commit_group;");
        };
        fill(kb0, 0);
        int stage = 0;
        for (int kb = kb0; kb <= k_hi; kb += 32, stage ^= 1) {
            fill(kb + 32, stage ^ 1);
            asm volatile("cp.async.wait_group 1;");
            __syncthreads();
            const float * ks = stages + (size_t) stage * 2 * 32 * kTileLd;
            const float * vs = ks + 32 * kTileLd;
            const bool here = good[stage][lane >> 2] >> (lane & 3) & 1;
            const int j = kb + lane;
            bool any = false;
#pragma unroll
            for (int i = 0; i < kWarpItems; i++) any |= kb <= last[i] && kb + 31 >= lo[i];
            if (any) {                                 // the same for all lanes: an item's numbers are the warp's
                unsigned long long dot[kWarpItems / 2];
#pragma unroll
                for (int pr = 0; pr < kWarpItems / 2; pr++) dot[pr] = 0ull;
                const float * kr = ks + lane * kTileLd;
                const float * qw = qs + (size_t) warp * kWarpItems * hd;
#pragma unroll 4
                for (int d = 0; d < hd; d += 4) {
                    const float4 k4 = *reinterpret_cast<const float4 *>(kr + d);
                    const unsigned long long k0 = pack2(k4.x, k4.x), k1 = pack2(k4.y, k4.y), k2 = pack2(k4.z, k4.z), k3 = pack2(k4.w, k4.w);
#pragma unroll
                    for (int pr = 0; pr < kWarpItems / 2; pr++) {
                        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(qw + (pr * hd + d) * 2);
                        const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(qw + (pr * hd + d + 2) * 2);
                        dot[pr] = fma2(a.x, k0, dot[pr]);
                        dot[pr] = fma2(a.y, k1, dot[pr]);
                        dot[pr] = fma2(b.x, k2, dot[pr]);
                        dot[pr] = fma2(b.y, k3, dot[pr]);
                    }
                }
                bool full = true;                      // every item weighs every key of the tile: no term is left out below
                float sc[kWarpItems], tile_max[kWarpItems], pj[kWarpItems], sum[kWarpItems], corr[kWarpItems];
                // step by step for all items, so that one's shuffles run in the shadow of another's; an item without a key here keeps
                // its maximum, and a factor of one and a sum of zero leave its numbers as they are
#pragma unroll
                for (int i = 0; i < kWarpItems; i++) {
                    const float2 two = unpack2(dot[i >> 1]);
                    const bool valid = here && j >= lo[i] && j <= last[i];
                    tile_max[i] = sc[i] = valid ? ((i & 1) ? two.y : two.x) * scale : -INFINITY;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < kWarpItems; i++) tile_max[i] = fmaxf(tile_max[i], __shfl_xor_sync(0xffffffffu, tile_max[i], o));
#pragma unroll
                for (int i = 0; i < kWarpItems; i++) {
                    const bool valid = here && j >= lo[i] && j <= last[i], some = tile_max[i] != -INFINITY;
                    const float m_new = fmaxf(m[i], tile_max[i]);
                    sum[i] = pj[i] = some && valid ? expf(sc[i] - m_new) : 0.0f;
                    corr[i] = !some ? 1.0f : m[i] == -INFINITY ? 0.0f : expf(m[i] - m_new);
                    if (some) m[i] = m_new;
                    full &= pj[i] != 0.0f;
                    ps[i * 32 + lane] = pj[i];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < kWarpItems; i++) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
#pragma unroll
                for (int i = 0; i < kWarpItems; i++) {
                    l[i] = l[i] * corr[i] + sum[i];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const float2 v = unpack2(acc[i][e]);
                        acc[i][e] = pack2(v.x * corr[i], v.y * corr[i]);
                    }
                }
                full = __all_sync(0xffffffffu, full);
                __syncwarp();
                if (full && lane < pieces) {
#pragma unroll 2
                    for (int jj = 0; jj < 32; jj += 4) {
                        ulonglong2 v[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) v[u] = *reinterpret_cast<const ulonglong2 *>(vs + (jj + u) * kTileLd + lane * 4);
#pragma unroll
                        for (int i = 0; i < kWarpItems; i++) {
                            const float4 p4 = *reinterpret_cast<const float4 *>(ps + i * 32 + jj);
                            const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                const unsigned long long pp = pack2(p[u], p[u]);
                                acc[i][0] = fma2(pp, v[u].x, acc[i][0]);
                                acc[i][1] = fma2(pp, v[u].y, acc[i][1]);
                            }
                        }
                    }
                } else if (lane < pieces) {
#pragma unroll 2
                    for (int jj = 0; jj < 32; jj += 4) {
                        ulonglong2 v[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) v[u] = *reinterpret_cast<const ulonglong2 *>(vs + (jj + u) * kTileLd + lane * 4);
#pragma unroll
                        for (int i = 0; i < kWarpItems; i++) {
                            const float4 p4 = *reinterpret_cast<const float4 *>(ps + i * 32 + jj);
                            const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int u = 0; u < 4; u++)
                                if (p[u] != 0.0f) {
                                    const unsigned long long pp = pack2(p[u], p[u]);
                                    acc[i][0] = fma2(pp, v[u].x, acc[i][0]);
                                    acc[i][1] = fma2(pp, v[u].y, acc[i][1]);
                                }
                        }
                    }
                }
                __syncwarp();
            }
            __syncthreads();                           // everyone is done with this stage before it is filled again
        }
        asm volatile("cp.async.wait_group 0;");
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kWarpItems; i++) {
        const int item = warp * kWarpItems + i;
        if (item >= n_items || lane >= pieces) continue;
        const int t = t0 + item / G, h = kvh * G + item % G;
        const float inv = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;
        const float2 x = unpack2(acc[i][0]), y = unpack2(acc[i][1]);
        float4 v = make_float4(x.x * inv, x.y * inv, y.x * inv, y.y * inv);
        if (gate != nullptr) {
            const float * g = gate + (size_t) t * ld_gate + h * hd + lane * 4;
            v.x *= 1.0f / (1.0f + expf(-g[0]));
            v.y *= 1.0f / (1.0f + expf(-g[1]));
            v.z *= 1.0f / (1.0f + expf(-g[2]));
            v.w *= 1.0f / (1.0f + expf(-g[3]));
        }
        float * o = out + ((size_t) t * nh + h) * hd + lane * 4;
        *reinterpret_cast<float4 *>(o) = v;
    }
}

template <typename A>
static int launch_generic(const A * q, const A * k_cache, const A * v_cache, A * out, const int * positions, const int * seq_of_token,
                          const int * block_table, int max_blocks, const int * ctx_len, int N, int nh, int nkv, int hd, int page_size,
                          int num_pages, float scale, int window, const float * sink, const A * gate, long long ld_gate, int tile_tokens,
                          cudaStream_t stream) {
    const unsigned blocks = (unsigned) (((long long) N * nh + kGenWarps - 1) / kGenWarps);
    const bool vec = (size_t) hd * sizeof(A) % 16 == 0 && (uintptr_t) k_cache % 16 == 0;
    auto go = [&](auto nacc, auto v) {
        paged_attention_generic_kernel<A, decltype(nacc)::value, decltype(v)::value><<<blocks, kGenWarps * 32, 0, stream>>>(
            q, k_cache, v_cache, out, positions, seq_of_token, block_table, max_blocks, ctx_len, N, nh, nkv, hd, page_size, num_pages,
            scale, window, sink, gate, ld_gate, tile_tokens);
    };
    auto pick = [&](auto v) {
        if (hd <= 64) go(std::integral_constant<int, 2>(), v);
        else if (hd <= 128) go(std::integral_constant<int, 4>(), v);
        else if (hd <= 256) go(std::integral_constant<int, 8>(), v);
        else go(std::integral_constant<int, kGenMaxHeadDim / 32>(), v);
    };
    if (vec) pick(std::true_type());
    else pick(std::false_type());
    return iian_launch_status();
}

}  // namespace iian

using namespace iian;

// q: [N, nh, hd]; caches: [num_pages, nkv, page_size, hd]; out: [N, nh * hd];
// block_table: [S, max_blocks]; ctx_len may be null (then only causality bounds the keys).
// sink: f32 [nh] or null; gate: rows of nh * hd with row stride ld_gate, or null
IIAN_API int iian_paged_attention_sink(
    const void * q, const void * k_cache, const void * v_cache, void * out,
    const int * positions, const int * seq_of_token, const int * block_table, int max_blocks,
    const int * ctx_len, int act_dtype, int N, int nh, int nkv, int hd, int page_size, int num_pages,
    float scale, int window, const float * sink, const void * gate, long long ld_gate, cudaStream_t stream) {
    if (N <= 0) return IIAN_OK;
    if (hd <= 0 || hd > kGenMaxHeadDim || nkv <= 0 || nh % nkv != 0 || page_size <= 0) return IIAN_ERR_SHAPE;
    if (act_dtype == IIAN_BF16)
        return launch_generic((const __nv_bfloat16 *) q, (const __nv_bfloat16 *) k_cache, (const __nv_bfloat16 *) v_cache, (__nv_bfloat16 *) out,
                              positions, seq_of_token, block_table, max_blocks, ctx_len, N, nh, nkv, hd, page_size, num_pages, scale, window,
                              sink, (const __nv_bfloat16 *) gate, ld_gate, 0, stream);
    if (act_dtype != IIAN_F32) return IIAN_ERR_DTYPE;
    // neighbouring tokens of a request share their key tiles where the sizes allow it; what is left (tokens of many requests side by
    // side, as when decoding) goes to the kernel with a warp per item, which leaves the others out (8 heads of 64 on one KV head, eight
    // requests behind 1,500: 244 us, 848 when a tile walks its four requests in turn; 16 on 2 of 128: 734 and 1,027)
    const int group = nh / nkv;
    // the tiled kernel moves 16 bytes at once on all four sides; the other one reads q and writes out an entry at a time
    const uintptr_t all = (uintptr_t) q | (uintptr_t) k_cache | (uintptr_t) v_cache | (uintptr_t) out;
    int tile_tokens = 0;
    if (N >= kTileMinTokens && group <= 8 && kTileItems % group == 0 && hd <= kTileHeadDim && hd % 4 == 0 && all % 16 == 0 && nkv <= 65535) {
        tile_tokens = kTileItems / group;
        const cudaError_t e = cudaFuncSetAttribute(paged_attention_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kTileSmem);
        if (e != cudaSuccess) return 1000 + (int) e;
        paged_attention_tile_kernel<<<dim3((N + tile_tokens - 1) / tile_tokens, nkv), kTileWarps * 32, kTileSmem, stream>>>(
            (const float *) q, (const float *) k_cache, (const float *) v_cache, (float *) out, positions, seq_of_token, block_table,
            max_blocks, ctx_len, N, nh, nkv, hd, page_size, num_pages, scale, window, sink, (const float *) gate, ld_gate);
        const int rc = iian_launch_status();
        if (rc != IIAN_OK) return rc;
    }
    return launch_generic((const float *) q, (const float *) k_cache, (const float *) v_cache, (float *) out, positions, seq_of_token,
                          block_table, max_blocks, ctx_len, N, nh, nkv, hd, page_size, num_pages, scale, window, sink, (const float *) gate,
                          ld_gate, tile_tokens, stream);
}

IIAN_API int iian_paged_attention_generic(
    const void * q, const void * k_cache, const void * v_cache, void * out,
    const int * positions, const int * seq_of_token, const int * block_table, int max_blocks,
    const int * ctx_len, int act_dtype, int N, int nh, int nkv, int hd, int page_size, int num_pages,
    float scale, int window, cudaStream_t stream) {
    return iian_paged_attention_sink(q, k_cache, v_cache, out, positions, seq_of_token, block_table, max_blocks, ctx_len, act_dtype,
                                     N, nh, nkv, hd, page_size, num_pages, scale, window, nullptr, nullptr, 0, stream);
}
