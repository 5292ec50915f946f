// out[n, m] = sum_k x[n, k] * w[m, k]: the plain matrix product of the 32-bit path, and the
// fallback for element-type combinations the tensor-core kernels do not take.
//
// Four forms with the same bits: tiles of register blocks for steps of many rows, smaller tiles fed by a ring for a few hundred, a form
// that streams the weights for steps of few (all three: float32 operands with rows of whole 16-byte pieces), and the plain one for
// everything else.
//
// Weights are row-major [out_features, in_features] exactly as the file stores them, which is
// also the reference's layout (ggml_mul_mat(W, x) = W x, src/iian/graph.cpp:121-160).  Products
// and sums are float32 FMAs (no reduced-precision matrix mode); every output element adds its
// K products in the order k = 0, 1, 2, ..., so a row's result does not depend on how many other
// rows the batch has.
#include <algorithm>

#include "common.cuh"
#include "packed.cuh"

namespace iian {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const TX * __restrict__ x, const TW * __restrict__ w,
                                                        TO * __restrict__ out, int N, int M, int K) {
    __shared__ float xs[BK][BN + 4];
    __shared__ float ws[BK][BM + 4];
    const int tid = threadIdx.x;
    const int n0 = blockIdx.y * BN, m0 = blockIdx.x * BM;
    const int tx = tid % 16, ty = tid / 16;          // thread computes rows n0 + ty*4.., cols m0 + tx*4..
    const int lrow = tid / 4, lk = (tid % 4) * 4;    // loader: row of the tile, first k of 4
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int k = k0 + lk + e;
            const int n = n0 + lrow, m = m0 + lrow;
            xs[lk + e][lrow] = (n < N && k < K) ? to_f32(x[(size_t) n * K + k]) : 0.0f;
            ws[lk + e][lrow] = (m < M && k < K) ? to_f32(w[(size_t) m * K + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = xs[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int n = n0 + ty * 4 + i;
        if (n >= N) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int m = m0 + tx * 4 + j;
            if (m < M) out[(size_t) n * M + m] = from_f32<TO>(acc[i][j]);
        }
    }
}

// Tiles of TILE_N rows x TILE_M columns, a thread TN x TM of them (in blocks of 4 x 4), operands through two stages of shared
// memory that lie k by k ([BK][rows + 4]), the loads of the next AHEAD stages under way in registers while one is multiplied (one
// alone leaves the latency of memory between the stages of a CTA that has its SM to itself).
// What bounds it: the float32 pipes and the reads of shared memory beside them (at 8 x 8, 3 clocks for every 8 of packed
// multiply-adds).  The loader's 16-byte pieces along k are put down as four words in four rows, the column flipped by 8 in the upper
// half of a stage so that a warp's words fall into 32 banks.  2,048 x 6,144 x 4,096: 2,023 us (51 TFLOP/s; 4 x 4 blocks without
// packing 3,996 us).
template <int TILE_N, int TILE_M, int TN, int TM, int AHEAD, typename TO>
__global__ void __launch_bounds__((TILE_N / TN) * (TILE_M / TM))
gemm_tile_kernel(const float * __restrict__ x, const float * __restrict__ w, TO * __restrict__ out, int N, int M, int K) {
    constexpr int THREADS = (TILE_N / TN) * (TILE_M / TM), TX = TILE_M / TM;
    constexpr int LX = TILE_N * BK / 4 / THREADS, LW = TILE_M * BK / 4 / THREADS;        // 16-byte pieces a thread loads per stage
    static_assert(LX * THREADS * 4 == TILE_N * BK && LW * THREADS * 4 == TILE_M * BK && BK == 16, "whole pieces per thread");
    __shared__ __align__(16) float xs[2][BK][TILE_N + 4];
    __shared__ __align__(16) float ws[2][BK][TILE_M + 4];
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int n0 = blockIdx.y * TILE_N, m0 = blockIdx.x * TILE_M;
    unsigned long long acc[TN][TM / 2];
#pragma unroll
    for (int i = 0; i < TN; i++)
#pragma unroll
        for (int j = 0; j < TM / 2; j++) acc[i][j] = 0ull;
    float4 px[AHEAD][LX], pw[AHEAD][LW];
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto fetch = [&](int k0, float4 (&px)[LX], float4 (&pw)[LW]) {
        const int k = k0 + (tid & 3) * 4;                    // K is a multiple of 4: a piece lies inside or outside as a whole
#pragma unroll
        for (int i = 0; i < LX; i++) {
            const int n = n0 + (tid + i * THREADS) / 4;
            px[i] = n < N && k < K ? __ldg(reinterpret_cast<const float4 *>(x + (size_t) n * K + k)) : zero;
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int m = m0 + (tid + i * THREADS) / 4;
            pw[i] = m < M && k < K ? __ldg(reinterpret_cast<const float4 *>(w + (size_t) m * K + k)) : zero;
        }
    };
    auto put = [&](int stage, const float4 (&px)[LX], const float4 (&pw)[LW]) {
        const int kq = tid & 3, flip = (kq >> 1) * 8;
#pragma unroll
        for (int i = 0; i < LX; i++) {
            const int r = ((tid + i * THREADS) / 4) ^ flip;
            xs[stage][kq * 4][r] = px[i].x; xs[stage][kq * 4 + 1][r] = px[i].y;
            xs[stage][kq * 4 + 2][r] = px[i].z; xs[stage][kq * 4 + 3][r] = px[i].w;
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int r = ((tid + i * THREADS) / 4) ^ flip;
            ws[stage][kq * 4][r] = pw[i].x; ws[stage][kq * 4 + 1][r] = pw[i].y;
            ws[stage][kq * 4 + 2][r] = pw[i].z; ws[stage][kq * 4 + 3][r] = pw[i].w;
        }
    };
#pragma unroll
    for (int d = 0; d < AHEAD; d++) fetch(d * BK, px[d], pw[d]);
    put(0, px[0], pw[0]);
    __syncthreads();
    const int stages = (K + BK - 1) / BK;
    auto turn = [&](int s, float4 (&fx)[LX], float4 (&fw)[LW], const float4 (&nx)[LX], const float4 (&nw)[LW]) {
        const int cur = s & 1;
        if (s + AHEAD < stages) fetch((s + AHEAD) * BK, fx, fw);
#pragma unroll
        for (int k = 0; k < BK; k++) {
            const int flip = (k >> 3) * 8;
            float a[TN];
            unsigned long long b[TM / 2];
#pragma unroll
            for (int i = 0; i < TN / 4; i++)
                *reinterpret_cast<float4 *>(a + 4 * i) = *reinterpret_cast<const float4 *>(&xs[cur][k][(i * (TILE_N / (TN / 4)) + ty * 4) ^ flip]);
#pragma unroll
            for (int j = 0; j < TM / 4; j++)
                *reinterpret_cast<ulonglong2 *>(b + 2 * j) =
                    *reinterpret_cast<const ulonglong2 *>(&ws[cur][k][(j * (TILE_M / (TM / 4)) + tx * 4) ^ flip]);
#pragma unroll
            for (int i = 0; i < TN; i++) {
                const unsigned long long v = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TM / 2; j++) acc[i][j] = fma2(v, b[j], acc[i][j]);
            }
        }
        if (s + 1 < stages) put(cur ^ 1, nx, nw);            // the other stage: last read before the barrier that ended the turn before
        __syncthreads();
    };
    for (int s0 = 0; s0 < stages; s0 += AHEAD) {
#pragma unroll
        for (int d = 0; d < AHEAD; d++)
            if (s0 + d < stages) turn(s0 + d, px[d], pw[d], px[(d + 1) % AHEAD], pw[(d + 1) % AHEAD]);
    }
#pragma unroll
    for (int i = 0; i < TN; i++) {
        const int n = n0 + (i / 4) * (TILE_N / (TN / 4)) + ty * 4 + i % 4;
        if (n >= N) continue;
#pragma unroll
        for (int j = 0; j < TM / 2; j++) {
            const int m = m0 + (j / 2) * (TILE_M / (TM / 4)) + tx * 4 + (j % 2) * 2;
            const float2 v = unpack2(acc[i][j]);
            if (m < M) out[(size_t) n * M + m] = from_f32<TO>(v.x);
            if (m + 1 < M) out[(size_t) n * M + m + 1] = from_f32<TO>(v.y);
        }
    }
}

// Small tiles for steps whose large ones would leave SMs idle: a warp covers 4 TN rows x 8 TM columns, a CTA WY x WX warps.  Operands lie
// in shared memory as they do in memory, along k, so that they come by cp.async through a ring and nothing is turned around; a
// thread reads four k of a row at once.  The multiply-adds are single ones: packed ones want neighbours of one k side by side.
// Lanes are dealt so that neighbours share a row of one operand or of the other (bits 0 and 4 pick the row of x, bits 1 to 3 that of w):
// 16-byte reads then take 2 clocks a warp, 4 where equal addresses lie 8 lanes apart.  What bounds it: one warp a scheduler leaves
// the 4-clock chain and the reads' latency bare, more of them the dispatch of three-operand multiply-adds (41 clocks for 32).
template <int TN, int TM, int WY, int WX, int STAGES, int DEPTH, typename TO>
__global__ void __launch_bounds__(WY * WX * 32)
gemm_ring_kernel(const float * __restrict__ x, const float * __restrict__ w, TO * __restrict__ out, int N, int M, int K) {
    constexpr int TILE_N = 4 * TN * WY, TILE_M = 8 * TM * WX, THREADS = WY * WX * 32, LD = DEPTH + 4, PIECES = DEPTH / 4;
    constexpr int LOADS = (TILE_N + TILE_M) * PIECES / THREADS;
    static_assert(LOADS * THREADS == (TILE_N + TILE_M) * PIECES && THREADS % PIECES == 0, "whole pieces per thread");
    extern __shared__ __align__(16) float ring[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.y * TILE_N, m0 = blockIdx.x * TILE_M;
    const int turns = (K + DEPTH - 1) / DEPTH;
    auto fill = [&](int s) {
        if (s < turns) {
            const int at = tid % PIECES * 4, k = s * DEPTH + at; // K is a multiple of 4: a piece lies inside or outside as a whole
            float * to = ring + (s % STAGES) * (TILE_N + TILE_M) * LD + at;
#pragma unroll
            for (int i = 0; i < LOADS; i++) {
                const int r = (tid + i * THREADS) / PIECES;
                const bool is_x = r < TILE_N;
                const int g = is_x ? n0 + r : m0 + r - TILE_N;
                const bool in = k < K && g < (is_x ? N : M);
                copy16(to + r * LD, in ? (is_x ? x : w) + (size_t) g * K + k : x, in);
            }
        }
        asm volatile("cp.async.commit_group;");
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) fill(s);
    float acc[TN][TM];
#pragma unroll
    for (int i = 0; i < TN; i++)
#pragma unroll
        for (int j = 0; j < TM; j++) acc[i][j] = 0.0f;
    const int row = warp / WX * 4 * TN + ((lane & 1) | (lane >> 4) << 1), col = warp % WX * 8 * TM + ((lane >> 1) & 7);
    for (int s = 0; s < turns; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2));
        __syncthreads();                                     // this stage has landed for everyone; the one before has been read by everyone
        fill(s + STAGES - 1);
        const float * xr = ring + ((s % STAGES) * (TILE_N + TILE_M) + row) * LD;
        const float * wr = ring + ((s % STAGES) * (TILE_N + TILE_M) + TILE_N + col) * LD;
#pragma unroll
        for (int k = 0; k < DEPTH; k += 4) {
            float4 a[TN], b[TM];
#pragma unroll
            for (int i = 0; i < TN; i++) a[i] = *reinterpret_cast<const float4 *>(xr + i * 4 * LD + k);
#pragma unroll
            for (int j = 0; j < TM; j++) b[j] = *reinterpret_cast<const float4 *>(wr + j * 8 * LD + k);
#pragma unroll
            for (int i = 0; i < TN; i++)
#pragma unroll
                for (int j = 0; j < TM; j++) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TN; i++)
#pragma unroll
                for (int j = 0; j < TM; j++) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TN; i++)
#pragma unroll
                for (int j = 0; j < TM; j++) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TN; i++)
#pragma unroll
                for (int j = 0; j < TM; j++) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TN; i++) {
        const int n = n0 + row + 4 * i;
        if (n >= N) continue;
#pragma unroll
        for (int j = 0; j < TM; j++) {
            const int m = m0 + col + 8 * j;
            if (m < M) out[(size_t) n * M + m] = from_f32<TO>(acc[i][j]);
        }
    }
}

// Steps of few rows: the weights stream through a ring of shared-memory stages (cp.async, 128 of K per stage), TILE_M weight
// rows per CTA; a thread owns one weight row and every (128 / TILE_M)-th row of x, so that an output stays one chain over k.
// What bounds it: HBM where there are many weight rows (32 per CTA: four CTAs an SM hold some 130 KB in flight); with few (8 per
// CTA, so that every SM has some) the chain itself, 4 cycles per k.  1 x 151,936 x 4,096: 394 us (6.3 TB/s; the plain form 2,777 us);
// 2 x 1,024 x 3,072: 20 us (210 us).
constexpr int kRowsThreads = 128, kRowsK = 128, kRowsMax = 16;

template <int TILE_M, int STAGES, int PER, typename TO>
__global__ void __launch_bounds__(kRowsThreads)
gemm_rows_kernel(const float * __restrict__ x, const float * __restrict__ w, TO * __restrict__ out, int N, int M, int K) {
    constexpr int LD = kRowsK + 4, GROUPS = kRowsThreads / TILE_M;       // rows 4 banks apart: 16-byte reads of 8 lanes hit 32 banks
    extern __shared__ __align__(16) float ring[];
    const int stage_floats = (TILE_M + N) * LD;
    const int tid = threadIdx.x, m0 = blockIdx.x * TILE_M, m = tid % TILE_M, g = tid / TILE_M;
    const int turns = (K + kRowsK - 1) / kRowsK;
    auto fill = [&](int s) {
        if (s < turns) {
            float * to = ring + (s % STAGES) * stage_floats;
            const int k0 = s * kRowsK;
            for (int e = tid; e < (TILE_M + N) * (kRowsK / 4); e += kRowsThreads) {
                const int r = e / (kRowsK / 4), k = k0 + (e % (kRowsK / 4)) * 4;
                const bool is_w = r < TILE_M;
                const bool in = k < K && (!is_w || m0 + r < M);
                const float * from = is_w ? w + (size_t) (m0 + r) * K + k : x + (size_t) (r - TILE_M) * K + k;
                copy16(to + r * LD + (k - k0), in ? from : x, in);
            }
        }
        asm volatile("cp.async.commit_group;");
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) fill(s);
    float acc[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) acc[i] = 0.0f;
    for (int s = 0; s < turns; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2));
        __syncthreads();                                     // this stage has landed for everyone; the one before has been read by everyone
        fill(s + STAGES - 1);
        if (g < N) {
            const float * wr = ring + (s % STAGES) * stage_floats + m * LD;
            const float * xr = ring + (s % STAGES) * stage_floats + TILE_M * LD;
#pragma unroll 8
            for (int k = 0; k < kRowsK; k += 4) {
                const float4 b = *reinterpret_cast<const float4 *>(wr + k);
#pragma unroll
                for (int i = 0; i < PER; i++) {
                    const int n = min(g + i * GROUPS, N - 1);
                    const float4 a = *reinterpret_cast<const float4 *>(xr + n * LD + k);
                    acc[i] = fmaf(a.x, b.x, acc[i]);
                    acc[i] = fmaf(a.y, b.y, acc[i]);
                    acc[i] = fmaf(a.z, b.z, acc[i]);
                    acc[i] = fmaf(a.w, b.w, acc[i]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int n = g + i * GROUPS;
        if (n < N && m0 + m < M) out[(size_t) n * M + m0 + m] = from_f32<TO>(acc[i]);
    }
}

template <int TILE_N, int TILE_M, int TN, int TM, int AHEAD, typename TO>
static int launch_tile(const float * x, const float * w, TO * out, int N, int M, int K, cudaStream_t stream) {
    const dim3 grid((M + TILE_M - 1) / TILE_M, (N + TILE_N - 1) / TILE_N);
    gemm_tile_kernel<TILE_N, TILE_M, TN, TM, AHEAD, TO><<<grid, (TILE_N / TN) * (TILE_M / TM), 0, stream>>>(x, w, out, N, M, K);
    return iian_launch_status();
}

template <int TN, int TM, int STAGES, int DEPTH, typename TO>
static int launch_ring(const float * x, const float * w, TO * out, int N, int M, int K, cudaStream_t stream) {
    constexpr int TILE_N = 8 * TN, TILE_M = 16 * TM;         // two by two warps
    constexpr size_t smem = (size_t) STAGES * (TILE_N + TILE_M) * (DEPTH + 4) * sizeof(float);
    auto kernel = gemm_ring_kernel<TN, TM, 2, 2, STAGES, DEPTH, TO>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess) return 1000 + (int) e;
    const dim3 grid((M + TILE_M - 1) / TILE_M, (N + TILE_N - 1) / TILE_N);
    kernel<<<grid, 128, smem, stream>>>(x, w, out, N, M, K);
    return iian_launch_status();
}

template <int TILE_M, int STAGES, int PER, typename TO>
static int launch_rows(const float * x, const float * w, TO * out, int N, int M, int K, cudaStream_t stream) {
    const size_t smem = (size_t) STAGES * (TILE_M + N) * (kRowsK + 4) * sizeof(float);
    auto kernel = gemm_rows_kernel<TILE_M, STAGES, PER, TO>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        if (e != cudaSuccess) return 1000 + (int) e;
    }
    kernel<<<(M + TILE_M - 1) / TILE_M, kRowsThreads, smem, stream>>>(x, w, out, N, M, K);
    return iian_launch_status();
}

// Up to kRowsMax rows the streaming form; its CTAs own 32 weight rows where there are enough of them for every SM, 8 below
// (us: 2 x 6,144 x 1,024 14.3 against 16.5; 16 x 4,096 x 4,096 67 against 96; but 4 x 4,096 x 12,288 113 against 76, 12 x 1,024 x 1,024
// 18.7 against 10.8).  Above, the tile that makes the fullest SM finish first; us:
//   rows x columns x K     64 x 128   64 x 64 (8 x 4)   ring: 32 x 64   32 x 32   16 x 32   the plain form
//   301 x 4,096 x 1,024       108            87               78            82        99         156
//   301 x 1,024 x 2,048       127            76               76            56        58         157
//   301 x 6,144 x 1,024       109           119              105           115       136
//   301 x 1,024 x 3,072       185           129              111            82        84
//   17 x 4,096 x 1,024         65            39               25            15        16          74
//   17 x 1,024 x 2,048        130            78               50            28        23
//   120 x 1,024 x 2,048       130            78               52            29        31
//   1,024 x 4,096 x 4,096     775           727              781           930     1,070       1,548
//   256 x 4,096 x 1,024        70            64               70            82        84
//   1,024 x 1,024 x 3,072     189           177              189           223       234
//   2,048 x 6,144 x 4,096   2,023         2,107                                                3,996
template <typename TO>
static int launch_f32(const float * x, const float * w, TO * out, int N, int M, int K, cudaStream_t stream) {
    if (N <= kRowsMax) {
        if (M < (N > 8 ? 4096 : 6144)) return launch_rows<8, 6, 1, TO>(x, w, out, N, M, K, stream);
        if (N <= 4) return launch_rows<32, 3, 1, TO>(x, w, out, N, M, K, stream);
        return N <= 8 ? launch_rows<32, 3, 2, TO>(x, w, out, N, M, K, stream) : launch_rows<32, 3, 4, TO>(x, w, out, N, M, K, stream);
    }
    // us per 1,024 of K: `alone` for the first tile of an SM, `more` for each further one that runs beside it (up to `beside`), `then` for
    // those that wait for one of them to end
    auto cost = [&](int tn, int tm, double alone, double more, int beside, double then) {
        if ((N + tn - 1) / tn > 65535) return 1e30;          // more row tiles than a grid has (of 64 rows a call that comes here has not)
        const long long tiles = (long long) ((N + tn - 1) / tn) * ((M + tm - 1) / tm), further = (tiles - 1) / 148;
        return alone + more * (double) std::min<long long>(further, beside) + then * (double) std::max<long long>(further - beside, 0);
    };
    const double wide = cost(64, 128, 65.0, 43.0, 1, 43.0), even = cost(64, 64, 45.0, 13.5, 1, 26.0);
    const double half = cost(32, 64, 24.5, 12.0, 2, 14.8), small = cost(32, 32, 15.0, 7.7, 2, 9.2), least = cost(16, 32, 11.5, 4.1, 2, 5.5);
    const double best = std::min({wide, even, half, small, least});
    if (wide == best) return launch_tile<64, 128, 8, 8, 1, TO>(x, w, out, N, M, K, stream);
    if (even == best) return launch_tile<64, 64, 8, 4, 3, TO>(x, w, out, N, M, K, stream);
    if (half == best) return launch_ring<4, 4, 3, 32, TO>(x, w, out, N, M, K, stream);
    if (small == best) return launch_ring<4, 2, 4, 64, TO>(x, w, out, N, M, K, stream);
    return launch_ring<2, 2, 4, 32, TO>(x, w, out, N, M, K, stream);
}

template <typename TX, typename TW, typename TO>
static int launch(const void * x, const void * w, void * out, int N, int M, int K, cudaStream_t stream) {
    dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN);
    gemm_simt_kernel<TX, TW, TO><<<grid, 256, 0, stream>>>((const TX *) x, (const TW *) w, (TO *) out, N, M, K);
    return iian_launch_status();
}

}  // namespace iian

using namespace iian;

IIAN_API int iian_gemm_simt(const void * x, int x_dtype, const void * w, int w_dtype, void * out, int out_dtype,
                            int N, int M, int K, cudaStream_t stream) {
    if (N <= 0 || M <= 0) return IIAN_OK;
    if (K <= 0) return IIAN_ERR_SHAPE;
    if ((M + BM - 1) / BM > 2147483647 || (N + BN - 1) / BN > 65535) return IIAN_ERR_LIMIT;
    typedef __nv_bfloat16 bf;
    if (x_dtype == IIAN_F32 && w_dtype == IIAN_F32 && K % 4 == 0 && ((uintptr_t) x | (uintptr_t) w) % 16 == 0)
        return out_dtype == IIAN_F32 ? launch_f32((const float *) x, (const float *) w, (float *) out, N, M, K, stream)
             : out_dtype == IIAN_BF16 ? launch_f32((const float *) x, (const float *) w, (bf *) out, N, M, K, stream) : (int) IIAN_ERR_DTYPE;
    const int key = x_dtype * 4 + w_dtype * 2 + out_dtype;
    switch (key) {
        case 0: return launch<float, float, float>(x, w, out, N, M, K, stream);
        case 1: return launch<float, float, bf>(x, w, out, N, M, K, stream);
        case 2: return launch<float, bf, float>(x, w, out, N, M, K, stream);
        case 3: return launch<float, bf, bf>(x, w, out, N, M, K, stream);
        case 4: return launch<bf, float, float>(x, w, out, N, M, K, stream);
        case 5: return launch<bf, float, bf>(x, w, out, N, M, K, stream);
        case 6: return launch<bf, bf, float>(x, w, out, N, M, K, stream);
        case 7: return launch<bf, bf, bf>(x, w, out, N, M, K, stream);
    }
    return IIAN_ERR_DTYPE;
}
