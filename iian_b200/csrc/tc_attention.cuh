// What the tcgen05 attention kernels share: barriers, copies, products, tensor memory, and the order in which
// the row tiles of a step's requests are taken.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "packed.cuh"

namespace iian {

constexpr unsigned kAtSpinLimit = 4u * 1000u * 1000u;

__device__ __forceinline__ unsigned at_smem(const void * p) { return (unsigned) __cvta_generic_to_shared(p); }
__device__ __forceinline__ void at_mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void at_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void at_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool at_wait(unsigned bar, unsigned parity) {
    for (unsigned spin = 0; spin < kAtSpinLimit; spin++) {
        unsigned done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void at_tma_4d(unsigned dst, const CUtensorMap * map, int x, int y, int z, int w, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}
__device__ __forceinline__ void at_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void at_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void at_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void at_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void at_mma(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc,
                                       unsigned accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with the A operand in tensor memory (lane = row, 32-bit column = two consecutive bf16 along K)
__device__ __forceinline__ void at_mma_ts(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned idesc,
                                          unsigned accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void at_ld32(unsigned taddr, unsigned * r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void at_st32(unsigned taddr, const unsigned * r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
__device__ __forceinline__ void at_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void at_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float at_min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float at_tanh(float x) {      // 1 - 2 / (1 + e^2x), absolute error of a few 1e-7
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * 2.8853900817779268f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return fmaf(-2.0f, r, 1.0f);
}
__device__ __forceinline__ float at_max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float at_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Shared-memory matrix descriptor with 128-byte swizzle.  K-major operand (rows of 128 bytes along K, groups of
// 8 rows 1024 bytes apart): lbo unused, sbo = 1024.  MN-major operand (V: a key's row holds 64 values of the
// head, 8 keys make a 1024-byte swizzle atom): lbo = distance between the two halves of the head, sbo = 1024
// = the next 8 keys.  Addresses and offsets in units of 16 bytes.
__device__ __forceinline__ unsigned long long at_desc(unsigned addr, unsigned lbo_bytes, unsigned sbo_bytes) {
    unsigned long long d = 0;
    d |= (unsigned long long) ((addr & 0x3FFFF) >> 4);
    d |= (unsigned long long) ((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (unsigned long long) ((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= (unsigned long long) 1 << 46;
    d |= (unsigned long long) 2 << 61;
    return d;
}
// bf16 x bf16 -> f32, M x N tile; b_mn: the B operand is MN-major (else both are K-major)
__host__ __device__ constexpr unsigned at_idesc(int m, int n, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | ((unsigned) (n >> 3) << 17) | ((unsigned) (m >> 4) << 24);
}

// The row tile a CTA works on: of which request, its number there, and that request's numbers.
struct AtPlace { int s, tile, q0, q_len, ctx; };

// Which request and row tile the `unit`-th CTA works on: the row tiles of all requests in falling order of the keys they
// see, so that the longest walks start first and the short ones fill the gaps at the end (in the order of the grid the longest tiles of
// the last request or head began when the GPU was already running empty: 197 against 138 us for three portions, 1,361 tokens together,
// behind 200 to 6,000 cached ones, heads of 128).  A row tile of `rows` rows sees ceil((pos0 + last token + 1) / KEYS) key tiles, which
// grows with its number; the number of row tiles of a request that see L key tiles or more is a closed form, and a warp finds the L of the
// unit by bisection with its lanes over the requests -- to an eighth of the longest walk, which balances as well and takes three
// steps of some hundred cycles.  Where no request has more than one row tile the order of the batch, which needs no search, is kept if all
// CTAs fit at once (`single` 1) or the longest walk is no 1.75 times the mean (`single` 2; 68 portions of 30 tokens 37.9 us,
// ranked 43; 100 of them behind 0 to 4,000 tokens 256, in the batch's order 272).  A whole warp
// calls it.
template <int KEYS>
__device__ __forceinline__ bool at_row_tile(const int * __restrict__ cu_q, const int * __restrict__ ctx_len, int num_seqs, int single, int G,
                                            int rows, int unit, AtPlace & at) {
    auto place = [&](int s, int q0, int q_len, int ctx, int tile) {
        at.s = s; at.q0 = q0; at.q_len = q_len; at.ctx = ctx; at.tile = tile;
        return tile >= 0;
    };
    auto in_order = [&](int s, int before) {
        if (s >= num_seqs) return false;
        const int q0 = cu_q[s], q_len = cu_q[s + 1] - q0, ctx = ctx_len[s];
        return place(s, q0, q_len, ctx, (q_len * G + rows - 1) / rows - 1 - before);
    };
    if (num_seqs == 1) return in_order(0, unit);
    if (single == 1) return in_order(unit, 0);
    const int lane = threadIdx.x & 31;
    constexpr int HELD = 4;                                  // requests a lane holds: lane, lane + 32, ...; further ones are read again
    auto request = [&](int i, int & len, int & pos0) {
        len = pos0 = 0;                                      // (none: no tokens, no row tiles)
        if (i < num_seqs) { len = cu_q[i + 1] - cu_q[i]; pos0 = max(ctx_len[i] - len, 0); }         // without context: sees no key, but is written
    };
    auto tiles_from = [&](int len, int pos0, int L) {        // row tiles of a request that see L key tiles or more
        const int n = (len * G + rows - 1) / rows, x = (L - 1) * KEYS - pos0;
        if (x <= 0) return n;
        return x < len ? n - x * G / rows : 0;               // the first of them holds row x * G
    };
    int len[HELD], pos0[HELD], all = 0, most = 0, sum = 0;
    auto add = [&](int q, int p) {
        all += tiles_from(q, p, 1);
        most = max(most, q > 0 ? p + q : 0);
        sum += p + q;
    };
#pragma unroll
    for (int h = 0; h < HELD; h++) request(lane + 32 * h, len[h], pos0[h]);
#pragma unroll
    for (int h = 0; h < HELD; h++) add(len[h], pos0[h]);
#pragma unroll 1
    for (int i = lane + 32 * HELD; i < num_seqs; i += 32) {
        int q, p;
        request(i, q, p);
        add(q, p);
    }
    all = __reduce_add_sync(0xffffffffu, all);
    most = __reduce_max_sync(0xffffffffu, most);
    if (single == 2) {
        sum = __reduce_add_sync(0xffffffffu, sum);
        if ((float) most * (float) (4 * num_seqs) < 7.0f * (float) sum) return in_order(unit, 0);
    }
    if (all <= unit) return false;
    const int step = (most + 8 * KEYS - 1) / (8 * KEYS);     // key tiles to an eighth
    int lo = 0, above = 0;                                   // row tiles that see 1 + step * lo or more > unit >= those of a higher eighth = above
#pragma unroll 1
    for (int bit = 4; bit > 0; bit >>= 1) {
        const int L = 1 + step * (lo | bit);
        int c = 0;
#pragma unroll
        for (int h = 0; h < HELD; h++)
            if (32 * h < num_seqs) c += tiles_from(len[h], pos0[h], L);
#pragma unroll 1
        for (int i = lane + 32 * HELD; i < num_seqs; i += 32) {
            int q, p;
            request(i, q, p);
            c += tiles_from(q, p, L);
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (c > unit) lo |= bit;
        else above = c;
    }
    int rest = unit - above;                                 // among the row tiles of this eighth, request by request
#pragma unroll 1
    for (int base = 0; base < num_seqs; base += 32) {
        int q, p;
        request(base + lane, q, p);
        const int more = tiles_from(q, p, 1 + step * (lo + 1)), c = tiles_from(q, p, 1 + step * lo) - more;
        int upto = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned here = __ballot_sync(0xffffffffu, upto > rest);
        if (here != 0) {
            const int l = __ffs(here) - 1, s = base + l;
            const int tile = __shfl_sync(0xffffffffu, (q * G + rows - 1) / rows - 1 - more - (rest - (upto - c)), l);
            return place(s, cu_q[s], __shfl_sync(0xffffffffu, q, l), ctx_len[s], tile);
        }
        rest -= __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// Row tiles a request may have, and those of a step: all together not more than N G / rows + S.
static inline long long at_tiles(int max_q_len, int G, int rows) { return ((long long) max_q_len * G + rows - 1) / rows; }
static inline long long at_units(int N, int S, int max_q_len, int G, int rows) {
    const long long each = at_tiles(max_q_len, G, rows) * S, all = (long long) N * G / rows + S;
    return each < all ? each : all;
}
// `single` of at_row_tile for a step whose row tiles are `copies` CTAs each, one CTA an SM
static inline int at_single(int N, int S, int max_q_len, int G, int rows, int copies) {
    if (at_tiles(max_q_len, G, rows) > 1) return 0;
    return at_units(N, S, max_q_len, G, rows) * copies <= 148 ? 1 : 2;
}

typedef CUresult (*AtEncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                               const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static AtEncodeFn at_encode_fn() {
    static AtEncodeFn fn = nullptr;
    if (fn == nullptr) {
        void * p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (AtEncodeFn) p;
    }
    return fn;
}

}  // namespace iian
