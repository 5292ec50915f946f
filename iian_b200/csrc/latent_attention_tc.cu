// Attention over a cached low-rank latent (bfloat16) on the fifth-generation tensor cores: portions of prompts, and decoded tokens of
// models with many heads.
//
// As in latent_attention_mma.cu the rows of a product are (token, head) pairs: all heads of a token score the same cached rows
// (c_j, kr_j), and the values are the front of those rows.  Neighbouring rows of a request are neighbouring rows of q, so a CTA's 128 rows
// are one box.  The output is up to 512 wide and tensor memory holds 512 columns, so a CTA works on a SHARE of the values' columns, 256 at
// most: with rank 512 two CTAs form the scores of the same rows, each for its own half of the output.
//
// Per tile of 64 keys: S = Q K^T (128 x 64, accumulated over the width in chunks of 64 columns, each a 128-byte-swizzled box of
// a page's rows) and O += P V (P from tensor memory as the A operand; V is the MN-major B operand as TMA left the chunks of this CTA's
// share) are tcgen05.mma.  Shared memory holds two tiles of keys (147 KB at width 576) and the chunks of Q outside the share; Q's own four
// lie in the 128 columns of tensor memory that O (256) and two S (128) leave.  Of a tile of keys the chunks outside the share are
// refilled once its scores are formed, those of the share once its P V is.  While the softmax works on tile i the chunks outside the
// share are multiplied for tile i + 1, then P V of tile i, then the share's chunks; P lies in the columns its S came from.
// Roles: warps 0, 10, 11 TMA (a box of 16 rows takes a warp some 70 cycles to issue and a tile has 36: one warp alone was the
// bound), warp 1 lane 0 the products, warps 2..9 the softmax, two threads a row: each takes half of a tile's keys and half of
// O's columns, and they exchange their maxima through shared memory.
//
// What bounds it: the tensor pipe, 3,600 cycles a tile -- products 64 keys wide are held up by their A rows (64 cycles from shared
// memory, 50 from tensor memory, where the product itself takes 32), and 128 keys do not fit beside Q.  16 heads, rank 512 + 64: two
// portions of 334 and 1,003 tokens, 600 cached, 92 us (354 on mma.sync), a prompt of 2,048 tokens 141 us (582), rank 256 64 us (366);
// with one tile of keys and all of Q in shared memory the first of them took 171 us (load, scores, softmax and P V in a row).
//
// The softmax opens at the sink (a logit per head without key or value), masks by causality and window and keeps the exact running
// maximum, so that the largest weight is 1 and not rounded, and sums the rounded weights: 1,000 tokens are off by 0.00201 of float64,
// on mma.sync by 0.00202 (0.0022 with a maximum that moves only when it grew by 2^8).  Every wait on an mbarrier is bounded: a role that
// gives up records where in `status`, and the CTA comes to the common exit, where tensor memory is freed.
#include <cuda.h>

#include "common.cuh"
#include "latent_merge.cuh"
#include "tc_attention.cuh"

namespace iian {

constexpr int LT_ROWS = 128, LT_KEYS = 64, LT_CHUNK = 64, LT_SHARE = 256;
constexpr int LT_LOADERS = 3, LT_THREADS = 32 * (9 + LT_LOADERS), LT_HALF = LT_KEYS / 2;
constexpr int LT_Q_BYTES = LT_ROWS * 128, LT_K_BYTES = LT_KEYS * 128;      // a chunk of Q, of a tile of keys
constexpr int LT_OWN = LT_SHARE / LT_CHUNK;     // chunks of a share
constexpr unsigned LT_S = 256u, LT_Q = 384u;    // tensor-memory columns of the two S (and P) and of Q's own chunks; O lies from column 0 on

struct LatentTcParams {
    __nv_bfloat16 * out;            // [N, H, rank]
    float * part_o, * part_ml;      // gridDim.y > 1 parts of the keys: [N * H, parts, rank] unnormalised, [N * H, parts, 2] maximum and sum
    const __nv_bfloat16 * q;        // [N, H, width]
    const int * cu_q, * ctx_len, * block_table;
    const float * sink;             // [H] or null
    int * status;                   // {code, where}; zero before the launch
    int num_seqs, max_blocks, H, rank, width, page_size, num_pages, window;
    int single;                     // as at_row_tile has it
    float scale, scale_log2, sink_to_raw;
};

__device__ __forceinline__ void lt_tma_2d(unsigned dst, const CUtensorMap * map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

__device__ __forceinline__ void lt_st16(unsigned taddr, const unsigned * r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}

// REST: chunks outside the share (width / 64 - 4).  The chunks lie in shared memory with those first, then the share's.
template <int REST>
__global__ void __launch_bounds__(LT_THREADS, 1) latent_attention_tc_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const LatentTcParams p) {
    extern __shared__ __align__(1024) unsigned char lt_smem_raw[];
    unsigned char * smem = (unsigned char *) (((uintptr_t) lt_smem_raw + 1023) & ~(uintptr_t) 1023);
    __shared__ __align__(8) unsigned long long q_full, rest_full[2], rest_free[2], own_full[2], own_free[2], tail_full, s_full[2], p_full[2], o_done;
    __shared__ unsigned tmem_base_s;
    __shared__ float pair_s[2][LT_ROWS];                           // [half][row]: maxima, at the end the sums

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int CHUNKS = REST + LT_OWN;
    const int shares = p.rank / LT_SHARE;
    const int H = p.H;
    AtPlace at;
    if (!at_row_tile<LT_KEYS>(p.cu_q, p.ctx_len, p.num_seqs, p.single, H, LT_ROWS, (int) blockIdx.x / shares, at)) return;
    const int s = at.s, row_tile = at.tile;
    const int part = (int) blockIdx.x % shares;                    // this CTA's share of the values: chunks own .. own + LT_OWN - 1
    const int own = part * LT_OWN;
    auto column = [&](int slot) { return (slot >= REST ? own + slot - REST : slot < own ? slot : slot + LT_OWN) * LT_CHUNK; };
    const int q0 = at.q0, q_len = at.q_len, pos0 = at.ctx - q_len;
    const int rows_total = q_len * H, row0 = row_tile * LT_ROWS;
    const int k_lo = p.window > 0 ? max(0, pos0 + row0 / H - p.window + 1) : 0;
    const int k_hi = max(-1, pos0 + min(rows_total - 1, row0 + LT_ROWS - 1) / H);      // -1: rows without a key, one tile with nothing in it
    int tile_lo = k_lo / LT_KEYS, n_tiles = k_hi / LT_KEYS - tile_lo + 1;
    const int parts = (int) gridDim.y;
    if (parts > 1) {
        const int per = (n_tiles + parts - 1) / parts;
        tile_lo += (int) blockIdx.y * per;
        n_tiles = min(per, n_tiles - (int) blockIdx.y * per);
        if (n_tiles <= 0) {                                        // an empty part
            const size_t at = (size_t) q0 * H + row0;
            const int rows = min(LT_ROWS, rows_total - row0);
            for (int e = threadIdx.x; e < rows * LT_SHARE; e += blockDim.x)
                p.part_o[((at + e / LT_SHARE) * parts + blockIdx.y) * p.rank + part * LT_SHARE + e % LT_SHARE] = 0.0f;
            if (part == 0 && (int) threadIdx.x < rows)
                *reinterpret_cast<float2 *>(p.part_ml + ((at + threadIdx.x) * parts + blockIdx.y) * 2) = make_float2(-INFINITY, 0.0f);
            return;
        }
    }
    unsigned char * sK = smem;                                     // [2][CHUNKS][64 keys][128 B]
    unsigned char * sQ = sK + 2 * CHUNKS * LT_K_BYTES;             // [REST][128 rows][128 B]
    // rows of the last tile behind the newest key
    const int past = tile_lo + n_tiles - 1 == k_hi / LT_KEYS ? LT_KEYS - 1 - k_hi % LT_KEYS : 0;
    int * status = p.status;

    if (threadIdx.x == 0) {
        at_mbar_init(at_smem(&q_full), 9); at_mbar_init(at_smem(&tail_full), 2); at_mbar_init(at_smem(&o_done), 1);
        for (int b = 0; b < 2; b++) {
            at_mbar_init(at_smem(&rest_full[b]), 1); at_mbar_init(at_smem(&rest_free[b]), 1);
            at_mbar_init(at_smem(&own_full[b]), 2); at_mbar_init(at_smem(&own_free[b]), 1);
            at_mbar_init(at_smem(&s_full[b]), 1); at_mbar_init(at_smem(&p_full[b]), 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    at_fence_before();
    __syncthreads();
    at_fence_after();
    const unsigned tmem_base = tmem_base_s;

    if (warp == 0 || warp >= 10) {
        // ---- loaders: warp 0 the chunks outside the share, warps 10 and 11 half of the share's each; a lane a page of the tile, a box per
        // page and chunk; the block table is read a tile ahead ------------------------------------------------------------------
        const int ps = p.page_size, pages = LT_KEYS / ps;
        const int * bt = p.block_table + (size_t) s * p.max_blocks;
        const bool rest = warp == 0;
        const int first = rest ? 0 : REST + (warp - 10) * (LT_OWN / 2), last = rest ? REST : first + LT_OWN / 2;
        auto page_of = [&](int i) {                                // the lane's page of tile i, as the table has it
            const int j0 = (tile_lo + i) * LT_KEYS + lane * ps;
            return i < n_tiles && lane < pages && j0 <= k_hi ? __ldg(bt + j0 / ps) : -1;
        };
        if (rest && lane == 0) {
            at_expect_tx(at_smem(&q_full), (unsigned) (REST * LT_Q_BYTES));
            for (int c = 0; c < REST; c++) lt_tma_2d(at_smem(sQ + c * LT_Q_BYTES), &map_q, column(c), q0 * H + row0, at_smem(&q_full));
        }
        int page = page_of(0);
        for (int i = 0; i < (first < last ? n_tiles : 0); i++) {
            const int page_next = page_of(i + 1), b = i & 1;
            unsigned char * tile = sK + b * CHUNKS * LT_K_BYTES;
            const unsigned full = at_smem(rest ? &rest_full[b] : &own_full[b]);
            int good = 1;
            if (lane == 0) {
                if (i >= 2) good = at_wait(at_smem(rest ? &rest_free[b] : &own_free[b]), (unsigned) ((i - 2) >> 1) & 1u) ? 1 : 0;
                if (good) at_expect_tx(full, (unsigned) ((last - first) * LT_K_BYTES));
                else { status[0] = 1; status[1] = i; }
            }
            if (!__all_sync(0xffffffffu, good)) break;
            if (lane < pages) {
                const int y = (page >= 0 && page < p.num_pages ? page : p.num_pages) * ps;         // out of range: filled with zeros
                for (int c = first; c < last; c++) lt_tma_2d(at_smem(tile + c * LT_K_BYTES + lane * ps * 128), &map_k, column(c), y, full);
            }
            page = page_next;
            if (!rest && i == n_tiles - 1 && past > 0) {           // rows behind the newest key: whatever they hold must not meet P's zeros
                good = at_wait(full, (unsigned) (i >> 1) & 1u) ? 1 : 0;
                if (!good && lane == 0) { status[0] = 7; status[1] = i; }
                if (!__all_sync(0xffffffffu, good)) break;
                for (int c = first; c < last; c++)
                    for (int e = lane; e < past * 8; e += 32)
                        reinterpret_cast<uint4 *>(tile + c * LT_K_BYTES + (LT_KEYS - past) * 128)[e] = make_uint4(0u, 0u, 0u, 0u);
                at_fence_async_smem();
                __syncwarp();
                if (lane == 0) at_arrive(at_smem(&tail_full));
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---- products --------------------------------------------------------------------------------------------------
        constexpr unsigned idesc_qk = at_idesc(LT_ROWS, LT_KEYS, false);
        constexpr unsigned idesc_pv = at_idesc(LT_ROWS, LT_SHARE, true);
        const unsigned long long dq = at_desc(at_smem(sQ), 16, 1024), dk = at_desc(at_smem(sK), 16, 1024);
        const unsigned long long dv = at_desc(at_smem(sK + REST * LT_K_BYTES), LT_K_BYTES, 1024);
        if (!at_wait(at_smem(&q_full), 0u)) { status[0] = 2; status[1] = 0; goto done; }
        at_fence_after();
        auto rest_scores = [&](int i) {
            if constexpr (REST > 0) {
                const int b = i & 1;
                const unsigned ph = (unsigned) (i >> 1) & 1u, d = tmem_base + LT_S + (unsigned) (b * LT_KEYS);
                const unsigned long long dkb = dk + (unsigned long long) (b * CHUNKS * (LT_K_BYTES >> 4));
                // the columns held P of tile i - 2
                if (!at_wait(at_smem(&rest_full[b]), ph) || (i >= 2 && !at_wait(at_smem(&own_free[b]), ph ^ 1u))) {
                    status[0] = 3; status[1] = i;
                    return false;
                }
                at_fence_after();
#pragma unroll
                for (int k = 0; k < 4 * REST; k++)                 // 16 values per step: 32 bytes inside the swizzle atom
                    at_mma(d, dq + (unsigned long long) ((k >> 2) * (LT_Q_BYTES >> 4) + (k & 3) * 2),
                           dkb + (unsigned long long) ((k >> 2) * (LT_K_BYTES >> 4) + (k & 3) * 2), idesc_qk, k > 0 ? 1u : 0u);
                at_commit(at_smem(&rest_free[b]));
            }
            return true;
        };
        auto own_scores = [&](int i) {
            const int b = i & 1;
            const unsigned ph = (unsigned) (i >> 1) & 1u, d = tmem_base + LT_S + (unsigned) (b * LT_KEYS);
            const unsigned long long dkb = dk + (unsigned long long) (b * CHUNKS * (LT_K_BYTES >> 4));
            if (!at_wait(at_smem(&own_full[b]), ph) || (i == n_tiles - 1 && past > 0 && !at_wait(at_smem(&tail_full), 0u))) {
                status[0] = 8; status[1] = i;
                return false;
            }
            at_fence_after();
#pragma unroll
            for (int k = 0; k < 4 * LT_OWN; k++)                   // ... and 8 columns of Q
                at_mma_ts(d, tmem_base + LT_Q + (unsigned) (k * 8),
                          dkb + (unsigned long long) ((REST + (k >> 2)) * (LT_K_BYTES >> 4) + (k & 3) * 2), idesc_qk, REST > 0 || k > 0 ? 1u : 0u);
            at_commit(at_smem(&s_full[b]));
            return true;
        };
        if (!rest_scores(0) || !own_scores(0)) goto done;
        for (int i = 0; i < n_tiles; i++) {
            const int b = i & 1;
            if (i + 1 < n_tiles && !rest_scores(i + 1)) goto done;
            if (!at_wait(at_smem(&p_full[b]), (unsigned) (i >> 1) & 1u)) { status[0] = 4; status[1] = i; goto done; }
            at_fence_after();
            const unsigned long long dvb = dv + (unsigned long long) (b * CHUNKS * (LT_K_BYTES >> 4));
#pragma unroll
            for (int k = 0; k < LT_KEYS / 16; k++)                 // 16 keys per step: 8 columns of packed P, 16 key rows of V
                at_mma_ts(tmem_base, tmem_base + LT_S + (unsigned) (b * LT_KEYS + k * 8), dvb + (unsigned long long) (k * 16 * 128 / 16),
                          idesc_pv, (i > 0 || k > 0) ? 1u : 0u);
            at_commit(at_smem(&own_free[b]));
            if (i + 1 < n_tiles && !own_scores(i + 1)) goto done;
        }
        at_commit(at_smem(&o_done));
    } else if (warp >= 2) {
        // ---- softmax: two threads a row ----------------------------------------------------------------------------------
        const int qd = warp & 3, half = (warp - 2) >> 2, r_ = qd * 32 + lane, R = row0 + r_;
        const bool row_ok = R < rows_total;
        const int row_pos = pos0 + (row_ok ? R / H : 0);
        const unsigned lane_addr = (unsigned) (qd * 32) << 16, tO = tmem_base + lane_addr + (unsigned) (half * (LT_SHARE / 2));
        const float sl = p.scale_log2;
        // the two warps of 32 rows
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + qd) : "memory"); };
        // Q's own chunks into tensor memory: 32-bit columns of two neighbouring values
#pragma unroll 1
        for (int c = half * (LT_OWN / 2); c < (half + 1) * (LT_OWN / 2); c++) {
            unsigned w[32];
            const uint4 * src = reinterpret_cast<const uint4 *>(p.q + ((size_t) q0 * H + R) * p.width + (own + c) * LT_CHUNK);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const uint4 x = row_ok ? src[e] : make_uint4(0u, 0u, 0u, 0u);
                w[4 * e] = x.x; w[4 * e + 1] = x.y; w[4 * e + 2] = x.z; w[4 * e + 3] = x.w;
            }
            at_st32(tmem_base + LT_Q + lane_addr + (unsigned) (c * 32), w);
        }
        at_wait_st();
        at_fence_before();
        __syncwarp();
        if (lane == 0) at_arrive(at_smem(&q_full));
        float m_run = -INFINITY, l_run = 0.0f;                     // the maximum of both halves, the sum of the thread's own
        if (p.sink != nullptr && row_ok && blockIdx.y == 0) {      // the sink counts once
            m_run = p.sink[R % H] * p.sink_to_raw;
            l_run = half == 0 ? 1.0f : 0.0f;
        }
        // a wait that gave up is recorded and the walk goes on, so that neither of a pair waits for the other for good
        bool failed = false;
        for (int i = 0; i < n_tiles; i++) {
            const int key0 = (tile_lo + i) * LT_KEYS + half * LT_HALF;
            const unsigned tS = tmem_base + LT_S + lane_addr + (unsigned) ((i & 1) * LT_KEYS);
            if (!failed && !at_wait(at_smem(&s_full[i & 1]), (unsigned) (i >> 1) & 1u)) { status[0] = 5; status[1] = i; failed = true; }
            __syncwarp();
            at_fence_after();
            unsigned v[LT_HALF];
            at_ld32(tS + (unsigned) (half * LT_HALF), v);
            at_wait_ld();
            const int hi = row_ok ? min(LT_HALF - 1, row_pos - key0) : -1, lo = p.window > 0 ? max(0, row_pos - p.window + 1 - key0) : 0;
            if (!__all_sync(0xffffffffu, lo <= 0 && hi >= LT_HALF - 1)) {
#pragma unroll
                for (int j = 0; j < LT_HALF; j++)
                    if (j < lo || j > hi) v[j] = 0xff800000u;      // -inf
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < LT_HALF; j += 8)
#pragma unroll
                for (int e = 0; e < 4; e++) mx4[e] = at_max3(mx4[e], __uint_as_float(v[j + 2 * e]), __uint_as_float(v[j + 2 * e + 1]));
            float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            pair_sync();                                           // (the maxima of the tile before have been read)
            pair_s[half][r_] = mx;
            pair_sync();                                           // (behind it both halves of S are in registers: P may be written)
            mx = fmaxf(mx, pair_s[half ^ 1][r_]);
            float corr = 1.0f;
            bool moved = false;
            if (mx > m_run) {
                corr = m_run == -INFINITY ? 0.0f : at_exp2((m_run - mx) * sl);
                m_run = mx;
                moved = true;
            }
            const float neg = m_run == -INFINITY ? 0.0f : m_run * sl;
            const unsigned long long sl2 = pack2(sl, sl), neg2 = pack2(-neg, -neg);
            unsigned long long sum2[2] = {0ull, 0ull};
#pragma unroll
            for (int j = 0; j < LT_HALF; j += 4)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const unsigned long long t = fma2(pack2(__uint_as_float(v[j + 2 * e]), __uint_as_float(v[j + 2 * e + 1])), sl2, neg2);
                    float t0, t1;
                    unpack2(t, t0, t1);
                    __nv_bfloat162 h = __floats2bfloat162_rn(at_exp2(t0), at_exp2(t1));
                    const unsigned w = *reinterpret_cast<unsigned *>(&h);
                    // the weights as they are multiplied, so that their rounding weighs on both sides of the quotient
                    sum2[e] = add2(sum2[e], pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)));
                    v[(j >> 1) + e] = w;
                }
            float s0, s1, s2, s3;
            unpack2(sum2[0], s0, s1);
            unpack2(sum2[1], s2, s3);
            l_run = l_run * corr + ((s0 + s1) + (s2 + s3));
            lt_st16(tS + (unsigned) (half * (LT_HALF / 2)), v);    // P as bf16 pairs into the columns S came from (32 of its 64)
            if (i > 0 && __any_sync(0xffffffffu, moved)) {
                if (!failed && !at_wait(at_smem(&own_free[(i - 1) & 1]), (unsigned) ((i - 1) >> 1) & 1u)) { status[0] = 9; status[1] = i; failed = true; }
                __syncwarp();
                at_fence_after();
                const unsigned long long corr2 = pack2(corr, corr);
#pragma unroll 1
                for (int c0 = 0; c0 < LT_SHARE / 2; c0 += 64) {
                    unsigned o[64];
                    at_ld32(tO + (unsigned) c0, o);
                    at_ld32(tO + (unsigned) c0 + 32u, o + 32);
                    at_wait_ld();
#pragma unroll
                    for (int j = 0; j < 64; j += 2) {
                        float a, b;
                        unpack2(mul2(pack2(__uint_as_float(o[j]), __uint_as_float(o[j + 1])), corr2), a, b);
                        o[j] = __float_as_uint(a);
                        o[j + 1] = __float_as_uint(b);
                    }
                    at_st32(tO + (unsigned) c0, o);
                    at_st32(tO + (unsigned) c0 + 32u, o + 32);
                }
            }
            at_wait_st();
            at_fence_before();
            __syncwarp();
            if (lane == 0) at_arrive(at_smem(&p_full[i & 1]));
        }
        pair_sync();
        pair_s[half][r_] = l_run;
        pair_sync();
        l_run += pair_s[half ^ 1][r_];
        if (!failed && !at_wait(at_smem(&o_done), 0u)) { status[0] = 6; status[1] = n_tiles; }
        __syncwarp();
        at_fence_after();
        if (parts > 1) {
            const size_t at = ((size_t) q0 * H + R) * parts + blockIdx.y;
            if (row_ok && part == 0 && half == 0) *reinterpret_cast<float2 *>(p.part_ml + at * 2) = make_float2(m_run * p.scale, l_run);
            float * dst = p.part_o + at * p.rank + part * LT_SHARE + half * (LT_SHARE / 2);
#pragma unroll 1
            for (int c0 = 0; c0 < LT_SHARE / 2; c0 += 32) {
                unsigned o[32];
                at_ld32(tO + (unsigned) c0, o);
                at_wait_ld();
                if (row_ok) {
#pragma unroll
                    for (int e = 0; e < 32; e += 4) *reinterpret_cast<uint4 *>(dst + c0 + e) = make_uint4(o[e], o[e + 1], o[e + 2], o[e + 3]);
                }
            }
            goto done;
        }
        const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
        __nv_bfloat16 * dst = p.out + ((size_t) q0 * H + R) * p.rank + part * LT_SHARE + half * (LT_SHARE / 2);
#pragma unroll 1
        for (int c0 = 0; c0 < LT_SHARE / 2; c0 += 32) {
            unsigned o[32];
            at_ld32(tO + (unsigned) c0, o);
            at_wait_ld();
            if (row_ok) {
#pragma unroll
                for (int q8 = 0; q8 < 4; q8++) {
                    uint4 pk;
                    unsigned * w = &pk.x;
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(o[8 * q8 + 2 * e]) * inv, __uint_as_float(o[8 * q8 + 2 * e + 1]) * inv);
                        w[e] = *reinterpret_cast<unsigned *>(&h);
                    }
                    *reinterpret_cast<uint4 *>(dst + c0 + 8 * q8) = pk;
                }
            }
        }
    }
done:
    at_fence_before();
    __syncthreads();
    if (warp == 1) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ---- decoded tokens: the keys as the rows of the products ---------------------------------------------------------------
// A decoded token has its heads for rows, 16 or fewer, and would leave most of a row tile empty.  Here a tile of 128 keys is the M operand:
// S^T = K Q^T (128 keys x 16 heads), and with P^T [16 heads][128 keys] in shared memory O^T = V^T P^T, the rank in blocks of 128 rows,
// V^T the same chunks read MN-major.  Every cached row passes shared memory once, for all heads.
// P is held as two bfloat16 parts, the upper 16 bits of a weight and what they leave, which are 32 columns of one product where 16 would
// take as long.  With one part the outputs were further from 64 bits than those of mma.sync, whose parts of the keys have a largest
// weight of 1, and so an exact one, each (rank 512, 48 tokens behind 800 to 4,000: 0.00192 for 0.00189, of which 0.00166 are the result's own rounding).
// The tiles of all sequences lie end to end, and the CTAs, one an SM, take equal stretches of that line: a stretch may end inside a sequence
// (its part goes to scratch memory, slot sequence + CTA) and go on into the next ones.  latent_line_merge_kernel puts the parts together.
// Roles: warps 0..3 the softmax (a thread a key, all heads), warp 4 lane 0 the products, warps 5.. the copies: one for each pair of the
// latent's chunks of 64 values (a ring of five pairs), one for the rotated chunk and Q.  The first pair's and the rotated chunk's share of a
// tile's scores is formed in the shadow of the softmax in front of it.
// What bounds it: 68 products a tile of rank 512, some 100 cycles each however few the heads (128 rows of A from shared memory), and the
// softmax between them, 5 us for the 3.3 a tile takes to arrive; tiles ahead fetched into the L2 make it slower.  16 heads, rank 512, us
// with the merge, on mma.sync and here: 48 tokens behind 800 to 4,000 cached 78 and 62, 64 behind 4,000 114 and 96, 128 behind 4,000 212 and
// 164 (rank 256: 55 and 38, 83 and 62, 153 and 105); the CTA's set-up, its first tile and the merge are 20, so that fewer keys stay with
// mma.sync (32 behind 4,000 57 and 62, 64 behind 1,500 49 and 52).  With 32 heads the kernel above is faster.
constexpr int LL_KEYS = 128, LL_HEADS = 16, LL_SLOTS = 5;
constexpr int LL_CHUNK_BYTES = LL_KEYS * 128, LL_PAIR_BYTES = 2 * LL_CHUNK_BYTES;
constexpr unsigned LL_O = 64u;                  // tensor-memory columns: two S^T from 0 on, the blocks of O^T behind
constexpr int kLineCtas = 148;

struct LatentLineParams {
    __nv_bfloat16 * out;            // [N, H, rank]
    float * part_o, * part_ml;      // [S + CTAs, H, rank] unnormalised, [S + CTAs, H, 2] maximum and sum
    const int * cu_q, * ctx_len, * seq_of_token, * block_table;
    const float * sink;             // [H] or null
    int * status;
    int num_seqs, max_blocks, H, rank, page_size, num_pages, window;
    float scale, scale_log2, sink_to_raw;
};

// Key tiles of a sequence's one token (0: no token, or padding), its row of q and its first tile.
__device__ __forceinline__ int ll_tiles(const LatentLineParams & p, int s, int & q0, int & ctx, int & tile_lo) {
    q0 = p.cu_q[s];
    ctx = p.ctx_len[s];
    tile_lo = 0;
    if (p.cu_q[s + 1] <= q0 || ctx <= 0 || p.seq_of_token[q0] < 0) return 0;
    tile_lo = (p.window > 0 ? max(0, ctx - p.window) : 0) / LL_KEYS;
    return (ctx - 1) / LL_KEYS - tile_lo + 1;
}
// All tiles, and those in front of sequence `before`.  A whole warp calls it.
__device__ __forceinline__ int ll_total(const LatentLineParams & p, int before, int & ahead) {
    int all = 0, q0, ctx, lo;
    ahead = 0;
    for (int s = threadIdx.x & 31; s < p.num_seqs; s += 32) {
        const int n = ll_tiles(p, s, q0, ctx, lo);
        all += n;
        if (s < before) ahead += n;
    }
    ahead = __reduce_add_sync(0xffffffffu, ahead);
    return __reduce_add_sync(0xffffffffu, all);
}
__device__ __forceinline__ int ll_border(int total, int cta, int ctas) { return ctas > 0 ? (int) ((long long) total * cta / ctas) : 0; }
__device__ __forceinline__ int ll_cta_of(int total, int tile, int ctas) { return (int) (((long long) (tile + 1) * ctas - 1) / total); }

__device__ __forceinline__ void ll_ld16(unsigned taddr, unsigned * r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
// Sixteen values over the 32 lanes, reduced: the values a lane carries are halved with every exchange; lane l ends with value l >> 1.
template <typename F> __device__ __forceinline__ float ll_reduce(float * a, F f) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int half = LL_HEADS / 2, o = 16; half >= 1; half >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < half; j++) {
            const float give = up ? a[j] : a[j + half], keep = up ? a[j + half] : a[j];
            a[j] = f(keep, __shfl_xor_sync(0xffffffffu, give, o));
        }
    }
    return f(a[0], __shfl_xor_sync(0xffffffffu, a[0], 1));
}

template <int PAIRS>
__global__ void __launch_bounds__(32 * (6 + PAIRS), 1) latent_line_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const LatentLineParams p) {
    constexpr int N = LL_HEADS, CHUNKS = 2 * PAIRS + 1, ROPES = 2, Q_BYTES = N * 128, P_BYTES = 2 * N * 128;
    extern __shared__ __align__(1024) unsigned char lt_smem_raw[];
    unsigned char * sK = (unsigned char *) (((uintptr_t) lt_smem_raw + 1023) & ~(uintptr_t) 1023);     // [LL_SLOTS][2 chunks][128 keys][128 B]
    unsigned char * sR = sK + LL_SLOTS * LL_PAIR_BYTES;            // [ROPES][128 keys][128 B]
    unsigned char * sQ = sR + ROPES * LL_CHUNK_BYTES;              // [CHUNKS][N heads][128 B]
    unsigned char * sP = sQ + CHUNKS * Q_BYTES;                    // [2][high parts, low parts][N heads][64 keys]
    __shared__ __align__(8) unsigned long long pair_full[LL_SLOTS], pair_free[LL_SLOTS], rope_full[ROPES], rope_free[ROPES], q_full, q_free, s_full, p_full, o_done;
    __shared__ unsigned tmem_base_s;
    __shared__ __align__(16) float wm[2][4][N], wl[4][N];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this CTA's stretch of the line: from tile `off` of sequence s on, `left` tiles
    int s = 0, off = 0, left;
    {
        int none;
        const int total = ll_total(p, 0, none), ctas = min((int) gridDim.x, total), g0 = ll_border(total, blockIdx.x, ctas);
        if ((int) blockIdx.x >= ctas) return;                      // (with fewer tiles than CTAs, one each)
        left = ll_border(total, blockIdx.x + 1, ctas) - g0;
        int run = 0;
        for (int base = 0; base < p.num_seqs; base += 32) {
            int q0, ctx, lo, n = base + lane < p.num_seqs ? ll_tiles(p, base + lane, q0, ctx, lo) : 0, upto = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const unsigned here = __ballot_sync(0xffffffffu, run + upto > g0);
            if (here != 0) {
                const int l = __ffs(here) - 1;
                s = base + l;
                off = g0 - (run + __shfl_sync(0xffffffffu, upto - n, l));
                break;
            }
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (threadIdx.x == 0) {
        for (int b = 0; b < LL_SLOTS; b++) { at_mbar_init(at_smem(&pair_full[b]), 1); at_mbar_init(at_smem(&pair_free[b]), 1); }
        for (int b = 0; b < ROPES; b++) { at_mbar_init(at_smem(&rope_full[b]), 1); at_mbar_init(at_smem(&rope_free[b]), 1); }
        at_mbar_init(at_smem(&q_full), 1); at_mbar_init(at_smem(&q_free), 1);
        at_mbar_init(at_smem(&s_full), 1); at_mbar_init(at_smem(&p_full), 4); at_mbar_init(at_smem(&o_done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    at_fence_before();
    __syncthreads();
    at_fence_after();
    const unsigned tmem_base = tmem_base_s;
    int * status = p.status;

    // the stretch, sequence by sequence: body(segment, sequence, its row of q, context, first key tile of it here, tiles here, tiles in all)
    auto walk = [&](auto body) {
        int s_ = s, off_ = off, left_ = left;
        for (int seg = 0; left_ > 0 && s_ < p.num_seqs; s_++) {
            int q0, ctx, lo;
            const int all = ll_tiles(p, s_, q0, ctx, lo);
            if (all <= off_) { off_ = 0; continue; }
            const int n = min(all - off_, left_);
            if (!body(seg, s_, q0, ctx, lo + off_, n, all, off_)) return;
            seg++;
            left_ -= n;
            off_ = 0;
        }
    };

    if (warp >= 5) {
        // ---- copies: a lane a page of the tile (of a pair: one for each chunk), the block table read a tile ahead -----------------
        const int ps = p.page_size, pages = LL_KEYS / ps, pr = warp - 5;
        const bool pair = pr < PAIRS;
        const int per = pair ? 2 : 1, pg = lane % pages, half = lane / pages;
        const bool mine = lane < per * pages;
        int it = 0;                                                // tiles of this CTA so far
        walk([&](int seg, int s_, int q0, int ctx, int tile0, int n, int, int) {
            const int * bt = p.block_table + (size_t) s_ * p.max_blocks;
            auto page_of = [&](int t) {
                const int j0 = (tile0 + t) * LL_KEYS + pg * ps;
                return t < n && mine && j0 < ctx ? __ldg(bt + j0 / ps) : -1;
            };
            int page = page_of(0), good = 1;
            if (!pair) {                                           // Q of this sequence, once the scores of the one before are formed
                if (lane == 0) {
                    if (seg > 0) good = at_wait(at_smem(&q_free), (unsigned) (seg - 1) & 1u) ? 1 : 0;
                    if (good) {
                        at_expect_tx(at_smem(&q_full), (unsigned) (CHUNKS * Q_BYTES));
                        for (int c = 0; c < CHUNKS; c++) lt_tma_2d(at_smem(sQ + c * Q_BYTES), &map_q, c * 64, q0 * p.H, at_smem(&q_full));
                    } else { status[0] = 31; status[1] = seg; }
                }
                if (!__all_sync(0xffffffffu, good)) return false;
            }
            for (int t = 0; t < n; t++, it++) {
                const int page_next = page_of(t + 1);
                const int k = pair ? it * PAIRS + pr : it, ring = pair ? LL_SLOTS : ROPES, slot = k % ring, round = k / ring;
                const unsigned full = at_smem(pair ? &pair_full[slot] : &rope_full[slot]);
                if (lane == 0) {
                    if (round > 0) good = at_wait(at_smem(pair ? &pair_free[slot] : &rope_free[slot]), (unsigned) (round - 1) & 1u) ? 1 : 0;
                    if (good) at_expect_tx(full, (unsigned) (pair ? LL_PAIR_BYTES : LL_CHUNK_BYTES));
                    else { status[0] = 32; status[1] = it; }
                }
                if (!__all_sync(0xffffffffu, good)) return false;
                if (mine) {
                    const int y = (page >= 0 && page < p.num_pages ? page : p.num_pages) * ps;         // out of range: filled with zeros
                    unsigned char * to = (pair ? sK + slot * LL_PAIR_BYTES + half * LL_CHUNK_BYTES : sR + slot * LL_CHUNK_BYTES) + pg * ps * 128;
                    lt_tma_2d(at_smem(to), &map_k, (pair ? 2 * pr + half : 2 * PAIRS) * 64, y, full);
                }
                page = page_next;
            }
            return true;
        });
    } else if (warp == 4) {
        if (lane == 0) {
            // ---- products ------------------------------------------------------------------------------------------------------
            constexpr unsigned idesc_s = at_idesc(LL_KEYS, N, false), idesc_o = at_idesc(128, 2 * N, false) | (1u << 15);      // V^T: A is MN-major
            const unsigned long long dk = at_desc(at_smem(sK), 16, 1024), dr = at_desc(at_smem(sR), 16, 1024), dq = at_desc(at_smem(sQ), 16, 1024);
            const unsigned long long dv = at_desc(at_smem(sK), LL_CHUNK_BYTES, 1024), dp = at_desc(at_smem(sP), 16, 1024);
            int it = 0;
            walk([&](int seg, int, int, int, int, int n, int, int) {
                if (!at_wait(at_smem(&q_full), (unsigned) seg & 1u)) { status[0] = 33; status[1] = seg; return false; }
                // the scores of tile i: one pair of chunks, the rotated chunk
                auto pair_scores = [&](int i, int pr, bool opens) {
                    const int k_ = i * PAIRS + pr, slot = k_ % LL_SLOTS;
                    if (!at_wait(at_smem(&pair_full[slot]), (unsigned) (k_ / LL_SLOTS) & 1u)) { status[0] = 34; status[1] = i; return false; }
                    at_fence_after();
#pragma unroll
                    for (int k = 0; k < 8; k++)                    // 16 values per step: 32 bytes inside the swizzle atom
                        at_mma(tmem_base + (unsigned) ((i & 1) * N), dk + (unsigned long long) (slot * (LL_PAIR_BYTES >> 4) + (k >> 2) * (LL_CHUNK_BYTES >> 4) + (k & 3) * 2),
                               dq + (unsigned long long) ((2 * pr + (k >> 2)) * (Q_BYTES >> 4) + (k & 3) * 2), idesc_s, !opens || k > 0 ? 1u : 0u);
                    return true;
                };
                auto rope_scores = [&](int i) {
                    const int rs = i % ROPES;
                    if (!at_wait(at_smem(&rope_full[rs]), (unsigned) (i / ROPES) & 1u)) { status[0] = 35; status[1] = i; return false; }
                    at_fence_after();
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        at_mma(tmem_base + (unsigned) ((i & 1) * N), dr + (unsigned long long) (rs * (LL_CHUNK_BYTES >> 4) + k * 2),
                               dq + (unsigned long long) (2 * PAIRS * (Q_BYTES >> 4) + k * 2), idesc_s, 1u);
                    at_commit(at_smem(&rope_free[rs]));
                    return true;
                };
                // what of a tile is there before the tile in front of it has been let go: the first pair and the rotated chunk
                auto early = [&](int i) { return pair_scores(i, 0, true) && rope_scores(i); };
                if (!early(it)) return false;
                for (int t = 0; t < n; t++, it++) {
#pragma unroll 1
                    for (int pr = 1; pr < PAIRS; pr++)
                        if (!pair_scores(it, pr, false)) return false;
                    if (t == n - 1) at_commit(at_smem(&q_free));
                    at_commit(at_smem(&s_full));
                    if (t + 1 < n && !early(it + 1)) return false;          // in the shadow of this tile's softmax
                    if (!at_wait(at_smem(&p_full), (unsigned) it & 1u)) { status[0] = 36; status[1] = it; return false; }
                    at_fence_after();
#pragma unroll 1
                    for (int pr = 0; pr < PAIRS; pr++) {           // 16 keys per step: 16 rows of V, 32 bytes of P
                        const int slot = (it * PAIRS + pr) % LL_SLOTS;
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            at_mma(tmem_base + LL_O + (unsigned) (pr * 2 * N), dv + (unsigned long long) (slot * (LL_PAIR_BYTES >> 4) + k * 128),
                                   dp + (unsigned long long) ((k >> 2) * (P_BYTES >> 4) + (k & 3) * 2), idesc_o, t > 0 || k > 0 ? 1u : 0u);
                        at_commit(at_smem(&pair_free[slot]));
                    }
                    if (t == n - 1) at_commit(at_smem(&o_done));
                }
                return true;
            });
        }
    } else {
        // ---- softmax: a thread a key, all heads ------------------------------------------------------------------------------
        const int r = threadIdx.x;
        const unsigned lane_addr = (unsigned) (warp * 32) << 16, tS = tmem_base + lane_addr, tO = tS + LL_O;
        const float sl = p.scale_log2;
        auto group_sync = [&]() { asm volatile("bar.sync 1, 128;" ::: "memory"); };
        auto larger = [](float a, float b) { return fmaxf(a, b); };
        auto sum = [](float a, float b) { return a + b; };
        bool failed = false;                                       // a wait that gave up is recorded and the walk goes on
        int it = 0;
        walk([&](int seg, int s_, int q0, int ctx, int tile0, int n, int all, int first) {
            float m_run[N], l_run[N];                              // the maximum of all keys, the sum of the thread's own
#pragma unroll
            for (int h = 0; h < N; h++) {
                const bool with = p.sink != nullptr && first == 0 && h < p.H;          // the sink counts once
                m_run[h] = with ? p.sink[h] * p.sink_to_raw : -INFINITY;
                l_run[h] = with && r == 0 ? 1.0f : 0.0f;
            }
            const int lo = p.window > 0 ? ctx - p.window : 0;
            for (int t = 0; t < n; t++, it++) {
                const int key0 = (tile0 + t) * LL_KEYS, j = key0 + r;
                if (!failed && !at_wait(at_smem(&s_full), (unsigned) it & 1u)) { status[0] = 37; status[1] = it; failed = true; }
                __syncwarp();
                at_fence_after();
                unsigned v[N];
                ll_ld16(tS + (unsigned) ((it & 1) * N), v);
                at_wait_ld();
                const bool seen = j < ctx && j >= lo;
                float a[N];
#pragma unroll
                for (int h = 0; h < N; h++) {
                    if (!seen) v[h] = 0xff800000u;                 // -inf
                    a[h] = __uint_as_float(v[h]);
                }
                const float mx = ll_reduce(a, larger);
                if ((lane & 1) == 0) wm[it & 1][warp][lane >> 1] = mx;
                // rows behind the newest key: whatever they hold must not meet P's zeros (pages without a key came as zeros)
                const int past = ctx - key0;
                if (past < LL_KEYS && r >= past) {
                    for (int pr = 0; pr < PAIRS; pr++) {
                        unsigned char * row = sK + (it * PAIRS + pr) % LL_SLOTS * LL_PAIR_BYTES + r * 128;
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            reinterpret_cast<uint4 *>(row)[e] = make_uint4(0u, 0u, 0u, 0u);
                            reinterpret_cast<uint4 *>(row + LL_CHUNK_BYTES)[e] = make_uint4(0u, 0u, 0u, 0u);
                        }
                    }
                }
                group_sync();
                // the exact running maximum, as above
                bool moved = false;
                float corr[N];
#pragma unroll
                for (int h = 0; h < N; h += 4) {
                    const float4 a0 = *reinterpret_cast<const float4 *>(&wm[it & 1][0][h]), a1 = *reinterpret_cast<const float4 *>(&wm[it & 1][1][h]);
                    const float4 a2 = *reinterpret_cast<const float4 *>(&wm[it & 1][2][h]), a3 = *reinterpret_cast<const float4 *>(&wm[it & 1][3][h]);
                    const float top[4] = {fmaxf(at_max3(a0.x, a1.x, a2.x), a3.x), fmaxf(at_max3(a0.y, a1.y, a2.y), a3.y),
                                          fmaxf(at_max3(a0.z, a1.z, a2.z), a3.z), fmaxf(at_max3(a0.w, a1.w, a2.w), a3.w)};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        corr[h + e] = 1.0f;
                        if (top[e] > m_run[h + e]) {
                            corr[h + e] = m_run[h + e] == -INFINITY ? 0.0f : at_exp2((m_run[h + e] - top[e]) * sl);
                            m_run[h + e] = top[e];
                            moved = true;
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < N; h += 2) {
                    float x[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const float neg = m_run[h + e] == -INFINITY ? 0.0f : m_run[h + e] * sl;
                        x[e] = at_exp2(fmaf(__uint_as_float(v[h + e]), sl, -neg));
                        l_run[h + e] = fmaf(l_run[h + e], corr[h + e], x[e]);
                    }
                    // two neighbouring keys in a word: the even lane takes head h, the odd one head h + 1
                    const bool odd = lane & 1;
                    const float got = __shfl_xor_sync(0xffffffffu, odd ? x[0] : x[1], 1), first_key = odd ? got : x[0], next_key = odd ? x[1] : got;
                    const unsigned b0 = __float_as_uint(first_key), b1 = __float_as_uint(next_key);
                    const int head = h + (odd ? 1 : 0), key = r & 62;
                    unsigned char * to = sP + (r >> 6) * P_BYTES + head * 128 + (((key >> 3) ^ (head & 7)) << 4) + (key & 7) * 2;
                    *reinterpret_cast<unsigned *>(to) = __byte_perm(b0, b1, 0x7632);
                    *reinterpret_cast<unsigned *>(to + N * 128) =
                        pack_bf16(first_key - __uint_as_float(b0 & 0xffff0000u), next_key - __uint_as_float(b1 & 0xffff0000u));
                }
                if (t > 0 && moved) {                              // (the scores of this tile followed the products of the one before)
#pragma unroll 1
                    for (int pr = 0; pr < PAIRS; pr++) {
                        unsigned o[2 * N];
                        at_ld32(tO + (unsigned) (pr * 2 * N), o);
                        at_wait_ld();
#pragma unroll
                        for (int h = 0; h < 2 * N; h++) o[h] = __float_as_uint(__uint_as_float(o[h]) * corr[h % N]);
                        at_st32(tO + (unsigned) (pr * 2 * N), o);
                    }
                    at_wait_st();
                }
                at_fence_async_smem();
                at_fence_before();
                __syncwarp();
                if (lane == 0) at_arrive(at_smem(&p_full));
            }
            // ---- this sequence's part ----------------------------------------------------------------------------------------
            const float mine = ll_reduce(l_run, sum);
            if ((lane & 1) == 0) wl[warp][lane >> 1] = mine;
            group_sync();
            if (!failed && !at_wait(at_smem(&o_done), (unsigned) seg & 1u)) { status[0] = 38; status[1] = it; failed = true; }
            __syncwarp();
            at_fence_after();
            const bool whole = n == all;
            const size_t slot = (size_t) s_ + blockIdx.x;
            float inv[N];
#pragma unroll
            for (int h = 0; h < N; h++) {
                const float l = (wl[0][h] + wl[1][h]) + (wl[2][h] + wl[3][h]);
                inv[h] = l > 0.0f ? 1.0f / l : 0.0f;
                if (!whole && r == 0 && h < p.H)
                    *reinterpret_cast<float2 *>(p.part_ml + (slot * p.H + h) * 2) = make_float2(m_run[h] * p.scale, l);
            }
#pragma unroll 1
            for (int pr = 0; pr < PAIRS; pr++) {
                unsigned o[2 * N];
                at_ld32(tO + (unsigned) (pr * 2 * N), o);
                at_wait_ld();
#pragma unroll
                for (int h = 0; h < N; h++) {
                    if (h >= p.H) continue;
                    const float both = __uint_as_float(o[h]) + __uint_as_float(o[h + N]);
                    if (whole) p.out[((size_t) q0 * p.H + h) * p.rank + pr * 128 + r] = __float2bfloat16_rn(both * inv[h]);
                    else p.part_o[(slot * p.H + h) * p.rank + pr * 128 + r] = both;
                }
            }
            group_sync();                                          // wl has been read
            return true;
        });
    }
    at_fence_before();
    __syncthreads();
    if (warp == 4) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(256u) : "memory");
    }
}

// Grid (S, H): the parts of a sequence that several CTAs walked; zeros for a token of no sequence.
__global__ void __launch_bounds__(128) latent_line_merge_kernel(const LatentLineParams p, int ctas) {
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, h = blockIdx.y;
    int q0, ctx, lo, ahead;
    const int n = ll_tiles(p, s, q0, ctx, lo);
    if (p.cu_q[s + 1] <= q0) return;
    __nv_bfloat16 * out = p.out + ((size_t) q0 * p.H + h) * p.rank;
    if (n == 0) {
        for (int c = threadIdx.x; c < p.rank; c += 128) out[c] = __float2bfloat16_rn(0.0f);
        return;
    }
    const int total = ll_total(p, s, ahead);
    ctas = min(ctas, total);
    const int first = ll_cta_of(total, ahead, ctas), last = ll_cta_of(total, ahead + n - 1, ctas);
    if (first == last) return;                                     // written whole
    const size_t slot = (size_t) s + first;
    float m = -INFINITY, l = 0.0f;
#pragma unroll 4
    for (int z = 0; z <= last - first; z++) m = fmaxf(m, p.part_ml[((slot + z) * p.H + h) * 2]);
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const int c = threadIdx.x * 4;
#pragma unroll 4
    for (int z = 0; z <= last - first; z++) {
        const float2 ml = *reinterpret_cast<const float2 *>(p.part_ml + ((slot + z) * p.H + h) * 2);
        const float w = ml.x == -INFINITY ? 0.0f : __expf(ml.x - m);
        l = fmaf(ml.y, w, l);
        if (c < p.rank) {
            const float4 x = *reinterpret_cast<const float4 *>(p.part_o + ((slot + z) * p.H + h) * p.rank + c);
            a[0] = fmaf(x.x, w, a[0]); a[1] = fmaf(x.y, w, a[1]); a[2] = fmaf(x.z, w, a[2]); a[3] = fmaf(x.w, w, a[3]);
        }
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
    if (c < p.rank) *reinterpret_cast<uint2 *>(out + c) = make_uint2(pack_bf16(a[0] * inv, a[1] * inv), pack_bf16(a[2] * inv, a[3] * inv));
}

// [rows, width] bf16, boxes of 64 columns x box_rows, 128-byte swizzle, zeros outside
static int lt_make_map(CUtensorMap * map, const void * base, long long rows, int width, int box_rows) {
    AtEncodeFn fn = at_encode_fn();
    if (fn == nullptr) return IIAN_ERR_LIMIT;
    cuuint64_t dims[2] = {(cuuint64_t) width, (cuuint64_t) rows};
    cuuint64_t strides[1] = {(cuuint64_t) width * 2};
    cuuint32_t box[2] = {LT_CHUNK, (cuuint32_t) box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? IIAN_OK : 2000 + (int) r;
}

template <int REST>
static int lt_launch(const CUtensorMap & mq, const CUtensorMap & mk, const LatentTcParams & p, dim3 grid, cudaStream_t stream) {
    const size_t smem = (size_t) REST * LT_Q_BYTES + (size_t) (REST + LT_OWN) * 2 * LT_K_BYTES + 1024;
    const cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel<REST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess) return 1000 + (int) e;
    latent_attention_tc_kernel<REST><<<grid, LT_THREADS, smem, stream>>>(mq, mk, p);
    return iian_launch_status();
}

template <int PAIRS>
static int ll_launch(const CUtensorMap & mq, const CUtensorMap & mk, const LatentLineParams & p, cudaStream_t stream) {
    const size_t smem = (size_t) LL_SLOTS * LL_PAIR_BYTES + 2 * LL_CHUNK_BYTES + (size_t) (2 * PAIRS + 5) * LL_HEADS * 128 + 1024;
    const cudaError_t e = cudaFuncSetAttribute(latent_line_kernel<PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess) return 1000 + (int) e;
    latent_line_kernel<PAIRS><<<kLineCtas, 32 * (6 + PAIRS), smem, stream>>>(mq, mk, p);
    return iian_launch_status();
}

}  // namespace iian

using namespace iian;

// 0 if the sizes are ones this kernel takes: rank 256 or 512, the row in chunks of 64 values (Q and a tile of keys must fit shared
// memory: width up to 576), pages of 8 to 64 tokens.
IIAN_API int iian_latent_attention_tc_ok(int rank, int width, int H, int page_size) {
    if ((rank != 256 && rank != 512) || width < rank || width % LT_CHUNK != 0 || width > 9 * LT_CHUNK || H <= 0) return IIAN_ERR_SHAPE;
    return page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64 ? IIAN_OK : IIAN_ERR_SHAPE;
}

// q: [N, H, width] bf16; cache: [num_pages * page_size, width] bf16; out: [N, H, rank] bf16; sink f32 [H] or null; scale > 0.
// parts (1..32): into how many parts the keys are cut; with more than one part_o [N * H, parts, rank] and part_ml [N * H, parts, 2] are needed.
// status: two ints on the device, zero before the launch; non-zero afterwards means a wait gave up and the output is not valid.
IIAN_API int iian_latent_attention_tc(const void * q, const void * cache, void * out, float * part_o, float * part_ml, const float * sink,
                                      const int * cu_q, const int * ctx_len, const int * seq_of_token, const int * block_table, int max_blocks,
                                      int N, int S, int max_q_len, int H, int rank, int width, int page_size, int num_pages, float scale, int window, int parts,
                                      int * status, cudaStream_t stream) {
    if (N <= 0 || S <= 0) return IIAN_OK;
    const int code = iian_latent_attention_tc_ok(rank, width, H, page_size);
    if (code != IIAN_OK) return code;
    if (!(scale > 0.0f) || status == nullptr || num_pages <= 0 || (long long) N * H < LT_ROWS) return IIAN_ERR_SHAPE;
    if (parts < 1 || parts > 32) return IIAN_ERR_SHAPE;
    if (parts > 1 && (part_o == nullptr || part_ml == nullptr || ((uintptr_t) part_o & 15) || ((uintptr_t) part_ml & 7))) return IIAN_ERR_SHAPE;
    if (((uintptr_t) q & 15) || ((uintptr_t) cache & 15) || ((uintptr_t) out & 15)) return IIAN_ERR_ALIGN;
    // a row number is a signed 32-bit coordinate of a copy
    if ((long long) N * H + LT_ROWS > 2147483647LL || (long long) (num_pages + 1) * page_size > 2147483647LL) return IIAN_ERR_LIMIT;
    CUtensorMap mq, mk;
    int rc = lt_make_map(&mq, q, (long long) N * H, width, LT_ROWS);
    if (rc != IIAN_OK) return rc;
    rc = lt_make_map(&mk, cache, (long long) num_pages * page_size, width, page_size);
    if (rc != IIAN_OK) return rc;
    LatentTcParams p;
    p.out = (__nv_bfloat16 *) out; p.q = (const __nv_bfloat16 *) q; p.part_o = part_o; p.part_ml = part_ml; p.scale = scale;
    p.cu_q = cu_q; p.ctx_len = ctx_len; p.block_table = block_table; p.sink = sink; p.status = status;
    p.num_seqs = S; p.max_blocks = max_blocks; p.H = H; p.rank = rank; p.width = width; p.page_size = page_size; p.num_pages = num_pages;
    p.window = window;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.sink_to_raw = 1.0f / scale;
    p.single = at_single(N, S, max_q_len, H, LT_ROWS, (rank / LT_SHARE) * parts);
    const dim3 grid((unsigned) (at_units(N, S, max_q_len, H, LT_ROWS) * (rank / LT_SHARE)), (unsigned) parts);
    int rc2 = IIAN_OK;
    switch (width / LT_CHUNK - LT_OWN) {
        case 0: rc2 = lt_launch<0>(mq, mk, p, grid, stream); break;
        case 1: rc2 = lt_launch<1>(mq, mk, p, grid, stream); break;
        case 2: rc2 = lt_launch<2>(mq, mk, p, grid, stream); break;
        case 3: rc2 = lt_launch<3>(mq, mk, p, grid, stream); break;
        case 4: rc2 = lt_launch<4>(mq, mk, p, grid, stream); break;
        default: rc2 = lt_launch<5>(mq, mk, p, grid, stream);
    }
    if (rc2 != IIAN_OK || parts == 1) return rc2;
    return latent_merge(part_o, part_ml, out, seq_of_token, N, H, parts, rank, stream);
}

// Decoded tokens (every sequence has one token at most), the keys as the rows of the products.  0 if the sizes are ones it takes: rank 256 or
// 512 with a rotated part of 64 values, 1 to 16 heads, pages of 8 to 128 tokens.
IIAN_API int iian_latent_line_ok(int rank, int width, int H, int page_size) {
    if ((rank != 256 && rank != 512) || width != rank + LT_CHUNK || H < 1 || H > LL_HEADS) return IIAN_ERR_SHAPE;
    return page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64 || page_size == 128 ? IIAN_OK : IIAN_ERR_SHAPE;
}
// Floats of scratch for a step of S sequences.
IIAN_API long long iian_latent_line_scratch(int S, int H, int rank) { return (long long) (S + kLineCtas) * H * (rank + 2); }

// As iian_latent_attention_tc; scratch: iian_latent_line_scratch floats on a 16-byte boundary.
IIAN_API int iian_latent_line(const void * q, const void * cache, void * out, float * scratch, const float * sink, const int * cu_q, const int * ctx_len,
                              const int * seq_of_token, const int * block_table, int max_blocks, int N, int S, int H, int rank, int width,
                              int page_size, int num_pages, float scale, int window, int * status, cudaStream_t stream) {
    if (N <= 0 || S <= 0) return IIAN_OK;
    const int code = iian_latent_line_ok(rank, width, H, page_size);
    if (code != IIAN_OK) return code;
    if (!(scale > 0.0f) || status == nullptr || num_pages <= 0 || scratch == nullptr) return IIAN_ERR_SHAPE;
    if (((uintptr_t) q & 15) || ((uintptr_t) cache & 15) || ((uintptr_t) out & 15) || ((uintptr_t) scratch & 15)) return IIAN_ERR_ALIGN;
    if (S > 65535 || (long long) N * H + 64 > 2147483647LL || (long long) (num_pages + 1) * page_size > 2147483647LL) return IIAN_ERR_LIMIT;
    if ((long long) N * H < LL_HEADS) return IIAN_ERR_SHAPE;           // a box of Q
    CUtensorMap mq, mk;
    int rc = lt_make_map(&mq, q, (long long) N * H, width, LL_HEADS);
    if (rc != IIAN_OK) return rc;
    rc = lt_make_map(&mk, cache, (long long) num_pages * page_size, width, page_size);
    if (rc != IIAN_OK) return rc;
    LatentLineParams p;
    p.out = (__nv_bfloat16 *) out;
    p.part_o = scratch; p.part_ml = scratch + (size_t) (S + kLineCtas) * H * rank;
    p.cu_q = cu_q; p.ctx_len = ctx_len; p.seq_of_token = seq_of_token; p.block_table = block_table; p.sink = sink; p.status = status;
    p.num_seqs = S; p.max_blocks = max_blocks; p.H = H; p.rank = rank; p.page_size = page_size; p.num_pages = num_pages; p.window = window;
    p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.sink_to_raw = 1.0f / scale;
    rc = rank == 512 ? ll_launch<4>(mq, mk, p, stream) : ll_launch<2>(mq, mk, p, stream);
    if (rc != IIAN_OK) return rc;
    return iian_launch(latent_line_merge_kernel, dim3((unsigned) S, (unsigned) H), dim3(128), 0, stream, p, kLineCtas);
}
