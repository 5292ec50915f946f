// The gated delta rule with a decay per key channel or per head: a recurrent mixer whose state is a matrix S [dim, vdim] per head.
//
// Per token and head, with unit vectors q (times dim^-1/2) and k, a value v, a write strength beta in (0, 1) and a decay
// g in (0, 1) per key channel (or one for the whole head: HEAD below):
//     S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// q, k and v come out of a short causal convolution over time (one filter per channel, the last tap is the current
// token's) followed by silu; the convolution's last `taps - 1` inputs are part of the state.
//
// The columns of S are independent: column j is a vector s_j of `dim` numbers with
//     s_j <- g * s_j;  u_j = beta (v_j - k . s_j);  s_j <- s_j + k u_j;  o_j = q . s_j = q . (g * s_j) + (q . k) u_j
// so a CTA owns kCols columns of one (sequence, head), kLanes lanes share a column (each holds every kLanes-th entry in
// registers), and both dot products of a token are taken from the decayed column in ONE pass and reduced together.
//
// Kernels:
//   delta_prep   per token and head: convolution + silu over the channels q | k | v (inputs of earlier tokens come from
//                the rows before it in the step, or from the state's tail), unit length of q and k per head, q . k, sigmoid
//                of the write strength, the decay exp(-exp(A) softplus(z + bias)).  Everything it leaves is float32.
//   delta_scan   the recurrence over a step's tokens of every sequence; the tokens' vectors come through two stages of
//                shared memory filled by cp.async a chunk ahead; the CTAs of a sequence also move the convolution's tail
//                on, a share of the channels each.
// With ONE decay per head the two dot products are taken from the column as it is and multiplied by the decay behind the
// reduction (g (k . s_j) = k . (g s_j)), so the multiplication of the column leaves the chain from token to token.
// State of a slot (float32): S as [heads, vdim, dim] (a column is contiguous), then the tail [taps - 1, channels].
#include <type_traits>

#include "common.cuh"
#include "packed.cuh"

namespace iian {

__device__ __forceinline__ float silu_f32(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f32(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

constexpr int kMaxTaps = 8;

// proj rows: [.. q (G * D) | k (G * D) | v (H * V) .. | b (H) ..] at col_off / b_off, row stride ld, activation type A.
// z: float32 rows of H * D, or of H with one decay per head (HEAD), row stride ld_z: the decay's pre-activation without its
// bias (dt_bias has as many numbers as a row).  b_pre: the write strengths' pre-activations in float32 (row stride ld_z), or
// null: the columns of proj at b_off.  taps: float32 [C, n_taps], C = 2 G D + H V.
// Grid (N, G + H): CTA (t, u) with u < G prepares query/key head u of token t (convolution, silu, unit length, q . k);
// with u >= G the values of head u - G (convolution, silu), that head's decays and its write strength -- so that a step of
// a few single tokens still spreads over the GPU.
constexpr int kPrepThreads = 128;
constexpr int kPrepMaxDim = 512;

template <typename A>
__device__ __forceinline__ float delta_conv(const A * __restrict__ proj, long long ld, int col, long long t, int first,
                                            const float * __restrict__ tail, int C, int c, const float * __restrict__ taps,
                                            int n_taps) {
    const int back = n_taps - 1;
    float x[kMaxTaps];
#pragma unroll
    for (int j = 0; j < kMaxTaps; j++) {
        x[j] = 0.0f;
        if (j < n_taps) {
            const long long r = t - back + j;                          // the row that tap j multiplies
            if (r >= first) x[j] = to_f32(proj[(size_t) r * ld + col]);
            else {
                const int idx = (int) (r - first) + back;              // place in the tail: rows first - back .. first - 1
                if (tail != nullptr && idx >= 0) x[j] = tail[(size_t) idx * C + c];
            }
        }
    }
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < kMaxTaps; j++)
        if (j < n_taps) acc = fmaf(taps[(size_t) c * n_taps + j], x[j], acc);
    return acc;
}

template <bool HEAD, typename A>
__global__ void __launch_bounds__(kPrepThreads)
delta_prep_kernel(const A * __restrict__ proj, long long ld, int col_off, int b_off, const float * __restrict__ b_pre,
                  const float * __restrict__ z, long long ld_z, const float * __restrict__ taps, int n_taps,
                  const float * __restrict__ a_log, const float * __restrict__ dt_bias,
                  const float * __restrict__ state, long long state_stride, long long tail_off,
                  const int * __restrict__ seq_of_token, const int * __restrict__ cu_q,
                  const int * __restrict__ state_slots,
                  float * __restrict__ qn, float * __restrict__ kn, float * __restrict__ vv,
                  float * __restrict__ beta, float * __restrict__ decay, float * __restrict__ qk,
                  int H, int G, int D, int V, float q_scale) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float act_q[kPrepMaxDim], act_k[kPrepMaxDim];
    __shared__ float red[3][kPrepThreads / 32];
    const size_t t = blockIdx.x;
    const int u = blockIdx.y;
    const int s = seq_of_token[t];
    const int GD = G * D, HV = H * V, C = 2 * GD + HV;
    if (s < 0) return;                         // padding token: the scan writes zeros for it
    const int slot = state_slots[s];
    const int first = cu_q[s];                 // the step's first row of this sequence
    const float * tail = slot >= 0 ? state + (size_t) slot * state_stride + tail_off : nullptr;
    if (u < G) {
        float sq = 0.0f, sk = 0.0f, dot = 0.0f;
        for (int d = threadIdx.x; d < D; d += kPrepThreads) {
            const int cq = u * D + d, ck = GD + u * D + d;
            const float a = silu_f32(delta_conv(proj, ld, col_off + cq, (long long) t, first, tail, C, cq, taps, n_taps));
            const float b = silu_f32(delta_conv(proj, ld, col_off + ck, (long long) t, first, tail, C, ck, taps, n_taps));
            act_q[d] = a;
            act_k[d] = b;
        }
        // the three sums in the order the tiled kernel takes them (a lane over d = lane, lane + 32, ..., then the lanes), so
        // that a token's vectors are the same bits whichever kernel prepared them
        __syncthreads();
        if (threadIdx.x < 32) {
            sq = sk = dot = 0.0f;
            for (int d = threadIdx.x; d < D; d += 32) {
                const float a = act_q[d], b = act_k[d];
                sq = fmaf(a, a, sq);
                sk = fmaf(b, b, sk);
                dot = fmaf(a, b, dot);
            }
            sq = warp_sum(sq);
            sk = warp_sum(sk);
            dot = warp_sum(dot);
            if (threadIdx.x == 0) { red[0][0] = sq; red[1][0] = sk; red[2][0] = dot; }
        }
        __syncthreads();
        sq = red[0][0]; sk = red[1][0]; dot = red[2][0];
        const float iq = q_scale / sqrtf(sq + 1e-6f), ik = 1.0f / sqrtf(sk + 1e-6f);
        for (int d = threadIdx.x; d < D; d += kPrepThreads) {
            qn[t * GD + u * D + d] = act_q[d] * iq;
            kn[t * GD + u * D + d] = act_k[d] * ik;
        }
        if (threadIdx.x == 0) qk[t * G + u] = dot * iq * ik;
        return;
    }
    const int h = u - G;
    for (int j = threadIdx.x; j < V; j += kPrepThreads) {
        const int c = 2 * GD + h * V + j;
        vv[t * HV + h * V + j] = silu_f32(delta_conv(proj, ld, col_off + c, (long long) t, first, tail, C, c, taps, n_taps));
    }
    const float rate = expf(a_log[h]);
    if (HEAD) {
        if (threadIdx.x == 0) decay[t * (size_t) H + h] = expf(-rate * softplus_f32(z[t * (size_t) ld_z + h] + dt_bias[h]));
    } else {
        for (int d = threadIdx.x; d < D; d += kPrepThreads) {
            const size_t e = (size_t) h * D + d;
            decay[t * (size_t) (H * D) + e] = expf(-rate * softplus_f32(z[t * (size_t) ld_z + e] + dt_bias[e]));
        }
    }
    if (threadIdx.x == 0) {
        const float zb = b_pre != nullptr ? b_pre[t * (size_t) ld_z + h] : to_f32(proj[t * ld + b_off + h]);
        beta[t * H + h] = 1.0f / (1.0f + expf(-zb));
    }
}

// The same preparation for steps of many tokens.  Grid (ceil(N / T), G + H): a CTA takes T neighbouring rows of the step for
// one unit (a query/key head, or a value head with its decays and write strength).  The rows the convolution needs
// (T + taps - 1 of them) and the unit's filters first go to shared memory, every load independent of the others, together with
// the tokens' sequence numbers; then each warp takes tokens of its own, a lane the entries lane, lane + 32, ...  Inputs from
// before a sequence's first row in the step come from the state's tail as in the kernel above.  Results are the same bits.
// Shared memory: x [T + taps - 1][W] rows of the unit's W channels | filters [taps][W] | first [T] | slot [T] (ints).
constexpr int kPrepTileWarps = 4;
constexpr int kPrepTileFrom = 256;          // tokens in a step from which the tiled kernel runs (tiles of 8; of 16 from four times as many)
constexpr int kPrepPerLane = kPrepMaxDim / 32;

template <bool HEAD, typename A>
__global__ void __launch_bounds__(kPrepTileWarps * 32)
delta_prep_tile_kernel(const A * __restrict__ proj, long long ld, int col_off, int b_off, const float * __restrict__ b_pre,
                       const float * __restrict__ z, long long ld_z, const float * __restrict__ taps, int n_taps,
                       const float * __restrict__ a_log, const float * __restrict__ dt_bias,
                       const float * __restrict__ state, long long state_stride, long long tail_off,
                       const int * __restrict__ seq_of_token, const int * __restrict__ cu_q,
                       const int * __restrict__ state_slots,
                       float * __restrict__ qn, float * __restrict__ kn, float * __restrict__ vv,
                       float * __restrict__ beta, float * __restrict__ decay, float * __restrict__ qk,
                       int N, int T, int H, int G, int D, int V, float q_scale) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) float psm[];
    const int u = blockIdx.y;
    const int GD = G * D, HV = H * V, C = 2 * GD + HV, HD = H * D;
    const int back = n_taps - 1, rows = T + back;
    const bool qk_unit = u < G;
    const int W = qk_unit ? 2 * D : V;                        // channels of this unit: q | k of a head, or a head's values
    float * xs = psm;                                        // [rows][W]
    float * ws = xs + (size_t) rows * W;                     // [n_taps][W]
    int * first_s = reinterpret_cast<int *>(ws + (size_t) W * n_taps);
    int * slot_s = first_s + T;
    const long long t0 = (long long) blockIdx.x * T;
    const int tid = threadIdx.x, nthr = blockDim.x;
    // channel w of the unit is channel chan(w) of the convolution
    auto chan = [&](int w) { return qk_unit ? (w < D ? u * D + w : GD + u * D + (w - D)) : 2 * GD + (u - G) * V + w; };
    if (tid < T) {
        const long long t = t0 + tid;
        int first = 0, slot = -2;                            // -2: no token (beyond the step, or padding)
        if (t < N) {
            const int sq = seq_of_token[t];
            if (sq >= 0) { first = cu_q[sq]; slot = state_slots[sq]; }
        }
        first_s[tid] = first;
        slot_s[tid] = slot;
    }
    for (int w = tid; w < W; w += nthr) {
        const int c = chan(w);
        const A * src = proj + col_off + c;
        for (int ri = 0; ri < rows; ri++) {
            const long long r = t0 - back + ri;
            xs[ri * W + w] = r >= 0 && r < N ? to_f32(src[(size_t) r * ld]) : 0.0f;
        }
        for (int j = 0; j < n_taps; j++) ws[j * W + w] = taps[(size_t) c * n_taps + j];      // [taps][W]: lanes read neighbours
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    // the convolution of channel w (convolution channel c) at the tile's token ti; `before` of its inputs lie ahead of the
    // sequence's first row in this step and come from the state's tail (or are zero)
    auto conv = [&](int ti, int before, const float * tail, int w, int c) {
        float acc = 0.0f;
        if (before <= 0) {
            for (int j = 0; j < n_taps; j++) acc = fmaf(ws[j * W + w], xs[(ti + j) * W + w], acc);
            return acc;
        }
        for (int j = 0; j < n_taps; j++) {
            float x = 0.0f;
            if (j >= before) x = xs[(ti + j) * W + w];
            else {
                const int idx = j - before + back;             // place in the tail: rows first - back .. first - 1
                if (tail != nullptr && idx >= 0) x = tail[(size_t) idx * C + c];
            }
            acc = fmaf(ws[j * W + w], x, acc);
        }
        return acc;
    };
    for (int ti = warp; ti < T; ti += kPrepTileWarps) {
        const int slot = slot_s[ti];
        if (slot == -2) continue;
        const long long t = t0 + ti;
        const int before = (int) (first_s[ti] - (t - back));        // inputs of this token that lie ahead of the step's rows
        const float * tail = slot >= 0 ? state + (size_t) slot * state_stride + tail_off : nullptr;
        if (qk_unit) {
            float aq[kPrepPerLane], ak[kPrepPerLane];
            float sq = 0.0f, sk = 0.0f, dot = 0.0f;
#pragma unroll
            for (int i = 0; i < kPrepPerLane; i++) {
                const int d = lane + 32 * i;
                aq[i] = ak[i] = 0.0f;
                if (d < D) {
                    aq[i] = silu_f32(conv(ti, before, tail, d, u * D + d));
                    ak[i] = silu_f32(conv(ti, before, tail, D + d, GD + u * D + d));
                    sq = fmaf(aq[i], aq[i], sq);
                    sk = fmaf(ak[i], ak[i], sk);
                    dot = fmaf(aq[i], ak[i], dot);
                }
            }
            sq = warp_sum(sq);
            sk = warp_sum(sk);
            dot = warp_sum(dot);
            const float iq = q_scale / sqrtf(sq + 1e-6f), ik = 1.0f / sqrtf(sk + 1e-6f);
#pragma unroll
            for (int i = 0; i < kPrepPerLane; i++) {
                const int d = lane + 32 * i;
                if (d < D) {
                    qn[t * GD + u * D + d] = aq[i] * iq;
                    kn[t * GD + u * D + d] = ak[i] * ik;
                }
            }
            if (lane == 0) qk[t * G + u] = dot * iq * ik;
        } else {
            const int h = u - G;
            const float rate = expf(a_log[h]);
            if (HEAD) {
                if (lane == 0) decay[t * (size_t) H + h] = expf(-rate * softplus_f32(z[t * (size_t) ld_z + h] + dt_bias[h]));
            } else {
                for (int d = lane; d < D; d += 32) {
                    const size_t e = (size_t) h * D + d;
                    decay[t * (size_t) HD + e] = expf(-rate * softplus_f32(z[t * (size_t) ld_z + e] + dt_bias[e]));
                }
            }
            for (int j = lane; j < V; j += 32)
                vv[t * HV + h * V + j] = silu_f32(conv(ti, before, tail, j, 2 * GD + h * V + j));
            if (lane == 0) {
                const float zb = b_pre != nullptr ? b_pre[t * (size_t) ld_z + h] : to_f32(proj[t * ld + b_off + h]);
                beta[t * H + h] = 1.0f / (1.0f + expf(-zb));
            }
        }
    }
}

// The same preparation for steps of many tokens of bfloat16 models with heads of 128 and four taps: a warp takes one unit of 128 channels
// (a query/key head's q and k, 128 values, a head's decays) over a few neighbouring rows, a lane four channels.  The
// convolution's window slides through registers, so every input is read once, four tokens ahead; nothing is staged
// and no lane waits for another but in the three sums of a query/key head.  There a lane has the channels lane, lane + 32, ... of the kernels
// above, so that the sums are taken in their order and the results are the same bits; values and decays go four neighbours a lane.
// What bounds it: instruction issue (the exponentials and
// logarithms of silu and softplus) and the latency of a window's loads.  1,500 tokens, 16 heads of 128 with a decay per channel: 35 us
// for 54 of the tiled kernel (replayed, the inputs in the L2; they and the results are 74 MB, 11 us).
constexpr int kWideWarps = 4;

template <bool HEAD, int kWideTokens>
__global__ void __launch_bounds__(kWideWarps * 32)
delta_prep_wide_kernel(const __nv_bfloat16 * __restrict__ proj, long long ld, int col_off, int b_off, const float * __restrict__ b_pre,
                       const float * __restrict__ z, long long ld_z, const float * __restrict__ taps,
                       const float * __restrict__ a_log, const float * __restrict__ dt_bias,
                       const float * __restrict__ state, long long state_stride, long long tail_off,
                       const int * __restrict__ seq_of_token, const int * __restrict__ cu_q, const int * __restrict__ state_slots,
                       float * __restrict__ qn, float * __restrict__ kn, float * __restrict__ vv,
                       float * __restrict__ beta, float * __restrict__ decay, float * __restrict__ qk,
                       int N, int H, int G, int V, float q_scale) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int D = 128, TAPS = 4, AHEAD = 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int GD = G * D, HV = H * V, C = 2 * GD + HV, v_units = HV / 128;
    const int t0 = blockIdx.x * kWideTokens, t1 = min(N, t0 + kWideTokens);
    const int u = blockIdx.y * kWideWarps + warp;
    if (u >= G + v_units + H) return;
    if (u >= G + v_units) {                      // decays and write strength of a head
        const int h = u - G - v_units;
        const float rate = expf(a_log[h]);
        if (HEAD) {                              // a lane is a token
            const int t = t0 + lane;
            if (lane < kWideTokens && t < t1 && seq_of_token[t] >= 0)
                decay[(size_t) t * H + h] = expf(-rate * softplus_f32(z[(size_t) t * ld_z + h] + dt_bias[h]));
        } else {
            const float4 bias = *reinterpret_cast<const float4 *>(dt_bias + h * D + 4 * lane);
#pragma unroll 4
            for (int t = t0; t < t1; t++) {
                const float4 x = *reinterpret_cast<const float4 *>(z + (size_t) t * ld_z + h * D + 4 * lane);
                float4 g;
                g.x = expf(-rate * softplus_f32(x.x + bias.x));
                g.y = expf(-rate * softplus_f32(x.y + bias.y));
                g.z = expf(-rate * softplus_f32(x.z + bias.z));
                g.w = expf(-rate * softplus_f32(x.w + bias.w));
                if (seq_of_token[t] >= 0) *reinterpret_cast<float4 *>(decay + (size_t) t * H * D + h * D + 4 * lane) = g;
            }
        }
        const int t = t0 + lane;
        if (lane < kWideTokens && t < t1 && seq_of_token[t] >= 0) {
            const float zb = b_pre != nullptr ? b_pre[(size_t) t * ld_z + h] : __bfloat162float(proj[(size_t) t * ld + b_off + h]);
            beta[(size_t) t * H + h] = 1.0f / (1.0f + expf(-zb));
        }
        return;
    }
    const bool is_qk = u < G;
    // this lane's channels, `apart` from one another: four of q and four of k, or four values
    const int c[2] = {is_qk ? u * D + lane : 2 * GD + (u - G) * 128 + 4 * lane, GD + u * D + lane};
    const int parts = is_qk ? 2 : 1, apart = is_qk ? 32 : 1;
    float w[2][4][TAPS], x[2][TAPS][4];          // filters; the last four inputs, the current one last
#pragma unroll
    for (int p = 0; p < 2; p++)
        if (p < parts)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float4 f = *reinterpret_cast<const float4 *>(taps + (size_t) (c[p] + e * apart) * TAPS);
                w[p][e][0] = f.x; w[p][e][1] = f.y; w[p][e][2] = f.z; w[p][e][3] = f.w;
            }
    auto input = [&](int p, long long r, float * to) {
        const __nv_bfloat16 * from = proj + (size_t) r * ld + col_off + c[p];
        if (is_qk) {
#pragma unroll
            for (int e = 0; e < 4; e++) to[e] = __bfloat162float(from[32 * e]);
            return;
        }
        const uint2 raw = *reinterpret_cast<const uint2 *>(from);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.y));
        to[0] = a.x; to[1] = a.y; to[2] = b.x; to[3] = b.y;
    };
    for (int tb = t0; tb < t1; tb += AHEAD) {
        float in[AHEAD][2][4];
        int sq[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            sq[i] = tb + i < t1 ? seq_of_token[tb + i] : -1;
#pragma unroll
            for (int p = 0; p < 2; p++)
                if (p < parts && tb + i < t1) input(p, tb + i, in[i][p]);
        }
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const int t = tb + i, s = sq[i];
            if (s < 0) continue;                 // padding, or behind the tile (the same for all lanes)
            const int first = cu_q[s];
            if (t == t0 || t == first || (i == 0 ? false : sq[i - 1] != s)) {       // the window anew: rows before t, or the state's tail
                const int slot = state_slots[s];
                const float * tail = slot >= 0 ? state + (size_t) slot * state_stride + tail_off : nullptr;
#pragma unroll
                for (int j = 1; j < TAPS; j++) {
                    const long long r = t - TAPS + j;                  // becomes the input of tap j - 1
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        if (p >= parts) continue;
                        if (r >= first) input(p, r, x[p][j]);
                        else {
                            const int idx = (int) (r - first) + TAPS - 1;
#pragma unroll
                            for (int e = 0; e < 4; e++) x[p][j][e] = tail != nullptr && idx >= 0 ? tail[(size_t) idx * C + c[p] + e * apart] : 0.0f;
                        }
                    }
                }
            }
            float a[2][4];
#pragma unroll
            for (int p = 0; p < 2; p++)
                if (p < parts)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        x[p][0][e] = x[p][1][e]; x[p][1][e] = x[p][2][e]; x[p][2][e] = x[p][3][e]; x[p][3][e] = in[i][p][e];
                        float acc = 0.0f;
#pragma unroll
                        for (int j = 0; j < TAPS; j++) acc = fmaf(w[p][e][j], x[p][j][e], acc);
                        a[p][e] = silu_f32(acc);
                    }
            if (!is_qk) {
                *reinterpret_cast<float4 *>(vv + (size_t) t * HV + c[0] - 2 * GD) = make_float4(a[0][0], a[0][1], a[0][2], a[0][3]);
                continue;
            }
            float s_q = 0.0f, s_k = 0.0f, dot = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s_q = fmaf(a[0][e], a[0][e], s_q);
                s_k = fmaf(a[1][e], a[1][e], s_k);
                dot = fmaf(a[0][e], a[1][e], dot);
            }
            s_q = warp_sum(s_q);
            s_k = warp_sum(s_k);
            dot = warp_sum(dot);
            const float iq = q_scale / sqrtf(s_q + 1e-6f), ik = 1.0f / sqrtf(s_k + 1e-6f);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                qn[(size_t) t * GD + c[0] + 32 * e] = a[0][e] * iq;
                kn[(size_t) t * GD + c[0] + 32 * e] = a[1][e] * ik;
            }
            if (lane == 0) qk[(size_t) t * G + u] = dot * iq * ik;
        }
    }
}

constexpr int kCols = 16;        // columns of S a CTA owns
constexpr int kLanes = 8;        // lanes that share a column

__device__ __forceinline__ void dr_cp4(float * dst, const float * src, bool valid) {
    const unsigned d = (unsigned) __cvta_generic_to_shared(dst);
    const int n = valid ? 4 : 0;                             // src-size 0: the word is zero-filled, nothing is read
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void dr_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void dr_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

// E: entries of a column a lane holds.  VEC (D a multiple of 4, the buffers 16-byte aligned): a lane holds groups of four
// neighbouring entries, d = 4 * lane + 32 * (i / 4) + i % 4, so that the state and the rows of q, k and the decays move
// 16 bytes at a time (E a multiple of 4); else entry d = lane + kLanes * i, word by word.  The tokens of a sequence pass
// through two stages of shared memory, `chunk` tokens each: while one is worked through, cp.async fills the other.
// HEAD: one decay per (token, head), decay [N, H]; it sits beside the write strength and q . k of its token.
// threads: those that call it (the launch's own number as a rule: with a constant, short portions take 2 to 4 percent longer).
__host__ __device__ constexpr int scan_floats(bool head, int Dp, int chunk) { return 2 * chunk * ((head ? 2 : 3) * Dp + kCols + 4); }      // of shared memory

template <int E, bool VEC, bool HEAD, typename A>
__device__ __forceinline__ void delta_scan(float * sm, const float * __restrict__ qn, const float * __restrict__ kn, const float * __restrict__ vv,
                  const float * __restrict__ beta, const float * __restrict__ decay, const float * __restrict__ qk,
                  float * __restrict__ state, long long state_stride, long long tail_off,
                  const A * __restrict__ proj, long long ld, int col_off, int n_taps,
                  const int * __restrict__ cu_q, const int * __restrict__ state_slots, float * __restrict__ out,
                  int H, int G, int D, int V, int chunk, unsigned threads) {
    const int Dp = (D + 3) & ~3;                             // rows start on 16-byte boundaries
    const int stage_floats = chunk * ((HEAD ? 2 : 3) * Dp + kCols + 4);      // q | k | decay (not HEAD) | v | beta, q . k, decay (HEAD), -
    const int cb = blockIdx.x, h = blockIdx.y, s = blockIdx.z;
    const int g = h / (H / G);
    const int col = threadIdx.x / kLanes, lane = threadIdx.x % kLanes;
    const int j = cb * kCols + col;            // this thread's column of S
    const int t0 = cu_q[s], t1 = cu_q[s + 1];
    const int slot = state_slots[s];
    const int HV = H * V, GD = G * D, HD = H * D;
    constexpr int kPer = HEAD ? 4 : 2;         // numbers per token behind the values
    if (slot < 0) {                            // a padding sequence: zeros out, nothing kept
        for (int t = t0; t < t1; t++)
            if (lane == 0 && j < V) out[(size_t) t * HV + h * V + j] = 0.0f;
        return;
    }
    float * st = state + (size_t) slot * state_stride;

    auto fill = [&](int c0, int stage) {       // tokens c0 .. of the step into a stage
        const int nt = min(chunk, t1 - c0);
        float * s_q = sm + (size_t) stage * stage_floats;
        float * s_k = s_q + chunk * Dp;
        float * s_g = s_k + chunk * Dp;
        float * s_v = s_g + (HEAD ? 0 : chunk * Dp);
        float * s_b = s_v + chunk * kCols;
        if (VEC) {
            const int per = D >> 2;
            for (int e = threadIdx.x; e < nt * per; e += threads) {
                const int tt = e / per, d = (e - tt * per) << 2;
                const size_t t = c0 + tt;
                copy16(s_q + tt * Dp + d, qn + t * GD + g * D + d);
                copy16(s_k + tt * Dp + d, kn + t * GD + g * D + d);
                if (!HEAD) copy16(s_g + tt * Dp + d, decay + t * HD + h * D + d);
            }
        } else {
            for (int e = threadIdx.x; e < nt * D; e += threads) {
                const int tt = e / D, d = e - tt * D;
                const size_t t = c0 + tt;
                dr_cp4(s_q + tt * Dp + d, qn + t * GD + g * D + d, true);
                dr_cp4(s_k + tt * Dp + d, kn + t * GD + g * D + d, true);
                if (!HEAD) dr_cp4(s_g + tt * Dp + d, decay + t * HD + h * D + d, true);
            }
        }
        for (int e = threadIdx.x; e < nt * kCols; e += threads) {
            const int tt = e / kCols, c = e - tt * kCols;
            const int jj = cb * kCols + c;
            dr_cp4(s_v + e, vv + (size_t) (c0 + tt) * HV + h * V + (jj < V ? jj : 0), jj < V);
        }
        for (int e = threadIdx.x; e < nt; e += threads) {
            dr_cp4(s_b + kPer * e, beta + (size_t) (c0 + e) * H + h, true);
            dr_cp4(s_b + kPer * e + 1, qk + (size_t) (c0 + e) * G + g, true);
            if (HEAD) dr_cp4(s_b + kPer * e + 2, decay + (size_t) (c0 + e) * H + h, true);
        }
    };
    if (t0 < t1) fill(t0, 0);
    dr_commit();

    // the convolution's tail moves on: the last taps - 1 inputs of the sequence so far (the sequence's CTAs share the channels)
    if (n_taps > 1) {
        const int C = 2 * GD + HV, back = n_taps - 1, L = t1 - t0;
        float * tail = st + tail_off;
        const int part = h * gridDim.x + cb, parts = gridDim.x * gridDim.y;
        for (int c = part * threads + threadIdx.x; c < C; c += parts * threads) {
            float keep[kMaxTaps];
#pragma unroll
            for (int i = 0; i < kMaxTaps - 1; i++) {
                if (i >= back) break;
                const int src = L - back + i;              // row of the step (relative to t0) that lands at place i
                keep[i] = src >= 0 ? to_f32(proj[(size_t) (t0 + src) * ld + col_off + c])
                                   : tail[(size_t) (src + back) * C + c];
            }
#pragma unroll
            for (int i = 0; i < kMaxTaps - 1; i++) {
                if (i >= back) break;
                tail[(size_t) i * C + c] = keep[i];
            }
        }
    }
    float S[E];
    float * scol = st + ((size_t) h * V + (j < V ? j : 0)) * D;
    static_assert(!VEC || E % 4 == 0, "groups of four entries");
    if (VEC) {
#pragma unroll
        for (int i = 0; i < E; i += 4) {
            const int d = 4 * lane + 4 * kLanes * (i >> 2);
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (j < V && d < D) x = *reinterpret_cast<const float4 *>(scol + d);
            S[i] = x.x; S[i + 1] = x.y; S[i + 2] = x.z; S[i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < E; i++) {
            const int d = lane + kLanes * i;
            S[i] = (j < V && d < D) ? scol[d] : 0.0f;
        }
    }
    int stage = 0;
    for (int c0 = t0; c0 < t1; c0 += chunk, stage ^= 1) {
        const int nt = min(chunk, t1 - c0);
        if (c0 + chunk < t1) {
            fill(c0 + chunk, stage ^ 1);       // (the stage was read two chunks ago; the barrier below closed that)
            dr_commit();
            dr_wait<1>();
        } else {
            dr_wait<0>();
        }
        __syncthreads();
        const float * s_q = sm + (size_t) stage * stage_floats;
        const float * s_k = s_q + chunk * Dp;
        const float * s_g = s_k + chunk * Dp;
        const float * s_v = s_g + (HEAD ? 0 : chunk * Dp);
        const float * s_b = s_v + chunk * kCols;
        for (int tt = 0; tt < nt; tt++) {
            const float * kq = s_k + tt * Dp;
            const float * qq = s_q + tt * Dp;
            const float * gg = s_g + tt * Dp;
            float a0 = 0.0f, a1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
            float kk[E];                       // the key's entries of this lane, kept for the write
            if (VEC) {
#pragma unroll
                for (int i = 0; i < E; i += 4) {
                    const int d = 4 * lane + 4 * kLanes * (i >> 2);
                    float4 g4 = make_float4(1.0f, 1.0f, 1.0f, 1.0f), k4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), q4 = k4;
                    if (d < D) {
                        if (!HEAD) g4 = *reinterpret_cast<const float4 *>(gg + d);
                        k4 = *reinterpret_cast<const float4 *>(kq + d);
                        q4 = *reinterpret_cast<const float4 *>(qq + d);
                    }
                    kk[i] = k4.x; kk[i + 1] = k4.y; kk[i + 2] = k4.z; kk[i + 3] = k4.w;
                    if (!HEAD) { S[i] *= g4.x; S[i + 1] *= g4.y; S[i + 2] *= g4.z; S[i + 3] *= g4.w; }
                    a0 = fmaf(k4.x, S[i], a0);     b0 = fmaf(q4.x, S[i], b0);
                    a1 = fmaf(k4.y, S[i + 1], a1); b1 = fmaf(q4.y, S[i + 1], b1);
                    a0 = fmaf(k4.z, S[i + 2], a0); b0 = fmaf(q4.z, S[i + 2], b0);
                    a1 = fmaf(k4.w, S[i + 3], a1); b1 = fmaf(q4.w, S[i + 3], b1);
                }
            } else {
#pragma unroll
                for (int i = 0; i < E; i += 2) {
                    const int d = lane + kLanes * i;
                    kk[i] = kk[i + 1] = 0.0f;
                    if (d < D) {
                        kk[i] = kq[d];
                        if (!HEAD) S[i] *= gg[d];
                        a0 = fmaf(kk[i], S[i], a0);
                        b0 = fmaf(qq[d], S[i], b0);
                    }
                    if (d + kLanes < D) {
                        kk[i + 1] = kq[d + kLanes];
                        if (!HEAD) S[i + 1] *= gg[d + kLanes];
                        a1 = fmaf(kk[i + 1], S[i + 1], a1);
                        b1 = fmaf(qq[d + kLanes], S[i + 1], b1);
                    }
                }
            }
            float a = a0 + a1, b = b0 + b1;
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, o);
                b += __shfl_xor_sync(0xffffffffu, b, o);
            }
            const float gd = HEAD ? s_b[kPer * tt + 2] : 1.0f;
            if (HEAD) { a *= gd; b *= gd; }
            const float u = s_b[kPer * tt] * (s_v[tt * kCols + col] - a);
#pragma unroll
            for (int i = 0; i < E; i++) S[i] = fmaf(kk[i], u, HEAD ? gd * S[i] : S[i]);     // (entries beyond D stay zero: their key is zero)
            if (lane == 0 && j < V) out[(size_t) (c0 + tt) * HV + h * V + j] = fmaf(s_b[kPer * tt + 1], u, b);
        }
        __syncthreads();                       // everyone is done with this stage before it is filled again
    }
    if (j < V) {
        if (VEC) {
#pragma unroll
            for (int i = 0; i < E; i += 4) {
                const int d = 4 * lane + 4 * kLanes * (i >> 2);
                if (d < D) *reinterpret_cast<float4 *>(scol + d) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int d = lane + kLanes * i;
                if (d < D) scol[d] = S[i];
            }
        }
    }
}

template <int E, bool VEC, bool HEAD, typename A>
__global__ void __launch_bounds__(kCols * kLanes)
delta_scan_kernel(const float * __restrict__ qn, const float * __restrict__ kn, const float * __restrict__ vv,
                  const float * __restrict__ beta, const float * __restrict__ decay, const float * __restrict__ qk,
                  float * __restrict__ state, long long state_stride, long long tail_off,
                  const A * __restrict__ proj, long long ld, int col_off, int n_taps,
                  const int * __restrict__ cu_q, const int * __restrict__ state_slots, float * __restrict__ out,
                  int H, int G, int D, int V, int chunk) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) float sm[];
    delta_scan<E, VEC, HEAD, A>(sm, qn, kn, vv, beta, decay, qk, state, state_stride, tail_off, proj, ld, col_off, n_taps, cu_q, state_slots, out,
                                H, G, D, V, chunk, blockDim.x);
}

// ---- portions of prompts, four tokens at a time ------------------------------------------------------------------
// Over four tokens the recurrence is a product with the state before them and small sums among themselves.  With G_t the decays'
// product from the first of the four to token t and G_ts that from the token behind s to t (both per key channel):
//     p_t = (G_t k_t) . s,  r_t = (G_t q_t) . s        eight dot products with ONE state column s
//     u_t = beta_t (v_t - p_t - sum_{s<t} A_ts u_s),   A_ts = sum_d k_t k_s G_ts
//     o_t = r_t + sum_{s<=t} B_ts u_s,                 B_ts = sum_d q_t k_s G_ts
//     s  <- G_3 s + sum_t (G_3t k_t) u_t
// so the chain from token to token (a pass over the column, a reduction over its lanes, the write) is walked once for four tokens.
// Everything is float32; the decays' products are of at most four factors, taken as such (no logarithms), and only ever shrink.
//   delta_block  per four tokens and head: the 13 vectors G_t k_t, G_t q_t, G_3t k_t, G_3 and the 28 numbers beta, A, B, one piece of
//                memory (tokens beyond a sequence's last count as k = q = 0, decay 1, beta 0: nothing changes).
//   delta_block_scan  the recurrence: the pieces come through a ring of four stages in shared memory, PER at a time.
constexpr int kBlockNumbers = 28;               // beta [4], A (1,0) (2,0) (2,1) (3,0) (3,1) (3,2) 0 0, B [4][4] (zero above the diagonal)
constexpr int kBlockStages = 4;

__device__ __forceinline__ float dr_both(unsigned long long v) {
    const float2 f = unpack2(v);
    return f.x + f.y;
}

// Where a sequence's pieces begin.  `pieces` 0: the whole step at once, the pieces of sequence s from cu_q[s] / 4 + s on (the sequences
// before it have no more: sum ceil(n / 4) <= floor(sum n / 4) + s); else the step in segments of that many pieces per sequence.
__device__ __forceinline__ size_t first_piece(const int * __restrict__ cu_q, int s, int pieces) {
    return pieces > 0 ? (size_t) s * pieces : (size_t) (cu_q[s] / 4 + s);
}

// Grid (all pieces, H) with the whole step at once, else (pieces of a segment, H, S); 128 threads; D <= 128.  Piece c of sequence s
// holds its tokens `from` + 4 c ..
__global__ void __launch_bounds__(128)
delta_block_kernel(const float * __restrict__ qn, const float * __restrict__ kn, const float * __restrict__ beta,
                   const float * __restrict__ decay, int per_head, const int * __restrict__ cu_q, const int * __restrict__ state_slots,
                   float * __restrict__ blocks, int from, int pieces, int at_least, int S, int H, int G, int D) {
    const int h = blockIdx.y, g = h / (H / G);
    int s = blockIdx.z, c = blockIdx.x;
    if (pieces == 0) {                           // the last sequence that begins at or before this piece
        int lo = 0, hi = S - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (cu_q[mid] / 4 + mid <= (int) blockIdx.x) lo = mid; else hi = mid - 1;
        }
        s = lo;
        c = (int) blockIdx.x - (cu_q[s] / 4 + s);
    }
    const long long t0 = (long long) cu_q[s] + from + 4 * c;
    const int n = (int) min(4ll, cu_q[s + 1] - t0);
    if (n <= 0 || state_slots[s] < 0 || cu_q[s + 1] - cu_q[s] < at_least) return;
    float * b = blocks + ((first_piece(cu_q, s, pieces) + c) * H + h) * (13 * D + kBlockNumbers);
    __shared__ float red[4][16];
    const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
    float k[4], q[4], w[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const bool in = t < n && d < D;
        const size_t row = (size_t) (t0 + t);
        k[t] = in ? kn[row * G * D + g * D + d] : 0.0f;
        q[t] = in ? qn[row * G * D + g * D + d] : 0.0f;
        w[t] = t < n ? (per_head ? decay[row * H + h] : d < D ? decay[row * H * D + h * D + d] : 1.0f) : 1.0f;
    }
    const float p0 = w[0], p1 = p0 * w[1], p2 = p1 * w[2], p3 = p2 * w[3];
    const float g21 = w[1] * w[2], g32 = w[2] * w[3], g31 = g21 * w[3];          // from the token behind 0 to 2, behind 1 to 3, behind 0 to 3
    if (d < D) {
        b[d] = p0 * k[0]; b[D + d] = p1 * k[1]; b[2 * D + d] = p2 * k[2]; b[3 * D + d] = p3 * k[3];
        b[4 * D + d] = p0 * q[0]; b[5 * D + d] = p1 * q[1]; b[6 * D + d] = p2 * q[2]; b[7 * D + d] = p3 * q[3];
        b[8 * D + d] = g31 * k[0]; b[9 * D + d] = g32 * k[1]; b[10 * D + d] = w[3] * k[2]; b[11 * D + d] = k[3];
        b[12 * D + d] = p3;
    }
    const float k0_1 = k[0] * w[1], k0_2 = k[0] * g21, k0_3 = k[0] * g31, k1_2 = k[1] * w[2], k1_3 = k[1] * g32, k2_3 = k[2] * w[3];
    float a[16] = {k[1] * k0_1, k[2] * k0_2, k[2] * k1_2, k[3] * k0_3, k[3] * k1_3, k[3] * k2_3,
                   q[0] * k[0], q[1] * k0_1, q[1] * k[1], q[2] * k0_2, q[2] * k1_2, q[2] * k[2],
                   q[3] * k0_3, q[3] * k1_3, q[3] * k2_3, q[3] * k[3]};
    // sixteen sums over the warp: the values a lane carries are halved with every exchange; a lane ends with value lane >> 1
#pragma unroll
    for (int half = 8; half >= 1; half >>= 1) {
        const bool up = lane & (2 * half);
#pragma unroll
        for (int j = 0; j < half; j++) {
            const float give = up ? a[j] : a[j + half], keep = up ? a[j + half] : a[j];
            a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * half);
        }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    if ((lane & 1) == 0) red[warp][lane >> 1] = a[0];
    __syncthreads();
    if (d < kBlockNumbers) {
        // place of each number among the sixteen sums; -1: zero, -2: a write strength
        const int from_sum[kBlockNumbers] = {-2, -2, -2, -2, 0, 1, 2, 3, 4, 5, -1, -1, 6, -1, -1, -1, 7, 8, -1, -1, 9, 10, 11, -1, 12, 13, 14, 15};
        int at = -1;
#pragma unroll
        for (int i = 0; i < kBlockNumbers; i++) at = i == d ? from_sum[i] : at;
        float v = 0.0f;
        if (at >= 0) v = (red[0][at] + red[1][at]) + (red[2][at] + red[3][at]);
        else if (at == -2 && d < n) v = beta[(size_t) (t0 + d) * H + h];
        b[13 * D + d] = v;
    }
}

// A CTA owns kCols columns of one (sequence, head); 16 lanes share two columns, E = D / 16 entries of each a lane (groups of four
// neighbours, d = 4 lane + 64 i): a vector that is read serves both.  Where the time goes: some 260 instructions a warp and piece with one
// warp per scheduler; of 920 clocks the eight dot products take 400, their reduction over the lanes 180, the four writes 170, the update 170,
// and shared memory's reads and shuffles fill 530 of them.
// AHEAD, where every CTA has an SM to itself: a fifth warp copies the pieces (350 clocks of a piece where every warp copied its share in its
// own chain), and their vectors are read into registers a step before they are needed; that takes 200 registers a thread, one CTA an SM, so
// it is not the form for more CTAs (32 heads, 2,048 tokens: 485 us in two rounds, 440 side by side).  1,500 tokens x 16 heads: 181 us (243
// without, with equal addresses 16 lanes apart; token by token 399).  Measured against the sixteen lanes: eight lanes a column, each
// column reading every vector for itself, 300 us (128 bytes a clock is what shared memory delivers to registers); 32 lanes for two columns, two
// warps per scheduler, 240 for then 256; a warp per eighth of D and a lane per column, the sums through shared memory, 241.
// V a multiple of kCols; state and values on 16-byte boundaries.
// Sequences with fewer than at_least tokens are walked token by token as in the scan above, in the same launch: a piece costs more than a
// token, and a launch of their own would wait for the long ones' chain (a portion of 100 tokens beside 100
// decoded ones, 16 heads with a decay per channel, through the mixer: 131 us, in two launches 166).  PER: pieces of a stage, 2 where the long
// walks decide, 1 where many short ones do, so that seven CTAs share an SM and not four (the same 131 us for 142, but 1,500 tokens 386 for 363);
// the launch bound asks for the registers that leaves (80 a thread are six CTAs: 100 portions of 40 tokens, 16 heads, 605 for 587).  With a decay a
// head the compiler finds them by itself, the thread count being a constant, and does better without the bound (562 for 554).
constexpr int kPairLanes = 16;

template <int E, int PER, bool AHEAD, bool HEAD, typename A>
__global__ void __launch_bounds__(kCols / 2 * kPairLanes + (AHEAD ? 32 : 0), PER == 1 && !HEAD ? 7 : 0)
delta_block_scan_kernel(const float * __restrict__ blocks, const float * __restrict__ qn, const float * __restrict__ kn,
                        const float * __restrict__ vv, const float * __restrict__ beta, const float * __restrict__ decay,
                        const float * __restrict__ qk, float * __restrict__ state, long long state_stride,
                        long long tail_off, const A * __restrict__ proj, long long ld, int col_off, int n_taps,
                        const int * __restrict__ cu_q, const int * __restrict__ state_slots, float * __restrict__ out,
                        int from, int pieces, int at_least, int H, int G, int V) {
    constexpr int D = E * kPairLanes, BLOCK = 13 * D + kBlockNumbers, PIECE = BLOCK + 4 * kCols, STAGE = PER * PIECE;
    constexpr int kThreads = kCols / 2 * kPairLanes;         // with AHEAD and a warp that copies
    constexpr bool EVERY = AHEAD || HEAD;
    extern __shared__ __align__(16) float sm[];
    const int cb = blockIdx.x, h = blockIdx.y, s = blockIdx.z;
    // neighbouring threads have the same entries of two pairs of columns: a 16-byte read then takes 2 clocks a warp, 4 where they lie 16 apart
    const int tid = threadIdx.x, pair = tid / 32 * 2 + (tid & 1), lane = tid % 32 >> 1, j = cb * kCols + 2 * pair;
    const int q0 = cu_q[s], q1 = cu_q[s + 1], slot = state_slots[s], HV = H * V;
    const int t0 = q0 + from, t1 = pieces > 0 ? min(q1, t0 + 4 * pieces) : q1;
    if (q1 - q0 < at_least) {
        constexpr int CHUNK = scan_floats(HEAD, D, 16) <= kBlockStages * STAGE ? 16 : 8;
        static_assert(kCols / 2 * kPairLanes == kCols * kLanes && scan_floats(HEAD, D, CHUNK) <= kBlockStages * STAGE, "both walks fit one launch");
        if (from == 0 && tid < kThreads)
            delta_scan<D / kLanes, true, HEAD, A>(sm, qn, kn, vv, beta, decay, qk, state, state_stride, tail_off, proj, ld, col_off, n_taps, cu_q,
                                                  state_slots, out, H, G, D, V, CHUNK, AHEAD || (HEAD && PER == 1) ? (unsigned) kThreads : blockDim.x);
        return;
    }
    if (t0 >= t1) return;
    if (slot < 0) {
        for (int t = t0; t < t1; t++)
            if (lane < 2 && tid < kThreads) out[(size_t) t * HV + h * V + j + lane] = 0.0f;
        return;
    }
    float * st = state + (size_t) slot * state_stride;
    const int n_blocks = (t1 - t0 + 3) / 4, turns = (n_blocks + PER - 1) / PER;
    const float * mine = blocks + (first_piece(cu_q, s, pieces) * H + h) * BLOCK;
    auto fill = [&](int turn, int me, auto threads) {
        constexpr int kCopiers = decltype(threads)::value;
        if (turn < turns) {
            float * to = sm + (turn % kBlockStages) * STAGE;
#pragma unroll
            for (int b = 0; b < PER; b++) {
                const int c = turn * PER + b;
                if (c >= n_blocks) break;
                const float * src = mine + (size_t) c * H * BLOCK;
#pragma unroll (kCopiers == 32 ? 4 : 1)
                for (int e = me; e < BLOCK / 4; e += kCopiers) copy16(to + b * PIECE + 4 * e, src + 4 * e);
                if (me < kCols) {                            // four tokens' values of the CTA's columns; beyond the last token: that one's
                    const int t = min(t0 + 4 * c + me / 4, t1 - 1);
                    copy16(to + b * PIECE + BLOCK + 4 * me, vv + (size_t) t * HV + h * V + cb * kCols + 4 * (me % 4));
                }
            }
        }
        dr_commit();
    };
    if constexpr (AHEAD) if (tid >= kThreads) {
        // The copying warp: every turn it waits for what is read next, and fills the stage that has been read by everyone.
        const std::integral_constant<int, 32> one_warp;
#pragma unroll
        for (int i = 0; i < kBlockStages - 1; i++) fill(i, tid - kThreads, one_warp);
        for (int turn = 0; turn < turns; turn++) {
            dr_wait<kBlockStages - 3>();
            __syncthreads();
            fill(turn + kBlockStages - 1, tid - kThreads, one_warp);
        }
        return;
    }
    const std::integral_constant<int, kThreads> all_warps;
    if constexpr (!AHEAD) {
#pragma unroll
        for (int i = 0; i < kBlockStages - 1; i++) fill(i, tid, all_warps);
    }

    if (from == 0 && n_taps > 1) {             // the convolution's tail moves on, as in the scan above
        const int C = 2 * G * D + HV, back = n_taps - 1, L = q1 - q0;
        float * tail = st + tail_off;
        const int part = h * gridDim.x + cb, parts = gridDim.x * gridDim.y;
        for (int c = part * kThreads + tid; c < C; c += parts * kThreads) {
            float keep[kMaxTaps];
#pragma unroll
            for (int i = 0; i < kMaxTaps - 1; i++) {
                if (i >= back) break;
                const int src = L - back + i;
                keep[i] = src >= 0 ? to_f32(proj[(size_t) (q0 + src) * ld + col_off + c]) : tail[(size_t) (src + back) * C + c];
            }
#pragma unroll
            for (int i = 0; i < kMaxTaps - 1; i++) {
                if (i >= back) break;
                tail[(size_t) i * C + c] = keep[i];
            }
        }
    }
    unsigned long long S[2][E / 2];
    float * scol = st + ((size_t) h * V + j) * D;
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
        for (int i = 0; i < E / 4; i++) {
            const ulonglong2 e = *reinterpret_cast<const ulonglong2 *>(scol + x * D + 4 * lane + 4 * kPairLanes * i);
            S[x][2 * i] = e.x; S[x][2 * i + 1] = e.y;
        }
    // AHEAD: a piece's vectors for the dot products are read while the piece before is reduced and written, from a stage that has landed a turn
    // early, and those for the update before the reduction, so that no read of shared memory stands in the chain.
    ulonglong2 dv[E / 4][8], uv[E / 4][5];
    float * to_out = out + (size_t) t0 * HV + h * V + j + (lane >> 3);
    auto piece = [&](int c) { return sm + (c / PER % kBlockStages) * STAGE + c % PER * PIECE; };
    auto at = [&](const float * vec, int v, int i) { return *reinterpret_cast<const ulonglong2 *>(vec + v * D + 4 * lane + 4 * kPairLanes * i); };
    auto read_dots = [&](const float * vec) {
#pragma unroll
        for (int i = 0; i < E / 4; i++)
#pragma unroll
            for (int v = 0; v < 8; v++) dv[i][v] = at(vec, v, i);
    };
    auto read_update = [&](const float * vec) {
#pragma unroll
        for (int i = 0; i < E / 4; i++)
#pragma unroll
            for (int v = 0; v < 5; v++) uv[i][v] = at(vec, 8 + v, i);
    };
    for (int turn = 0; turn < turns; turn++) {
        if (!AHEAD) dr_wait<kBlockStages - 2>();
        __syncthreads();                       // this turn's pieces have landed (and the next one's); the stage filled next was read by everyone
        if constexpr (!AHEAD) fill(turn + kBlockStages - 1, tid, all_warps);
        if (AHEAD && turn == 0) read_dots(piece(0));
#pragma unroll
        for (int b = 0; b < PER; b++) {
            const int c = turn * PER + b;
            if (c >= n_blocks) break;
            const float * vec = piece(c);
            const float * num = vec + 13 * D;
            unsigned long long acc[2][8];
#pragma unroll
            for (int v = 0; v < 8; v++) acc[0][v] = acc[1][v] = 0ull;
#pragma unroll
            for (int i = 0; i < E / 4; i++) {
#pragma unroll
                for (int v = 0; v < 8; v++) {
                    const ulonglong2 e = AHEAD ? dv[i][v] : at(vec, v, i);
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        acc[x][v] = fma2(e.x, S[x][2 * i], acc[x][v]);
                        acc[x][v] = fma2(e.y, S[x][2 * i + 1], acc[x][v]);
                    }
                }
            }
            const float4 be = *reinterpret_cast<const float4 *>(num), A0 = *reinterpret_cast<const float4 *>(num + 4);
            const float2 A1 = *reinterpret_cast<const float2 *>(num + 8);
            float4 B;
            if (EVERY) B = *reinterpret_cast<const float4 *>(num + 12 + 4 * (lane & 3));
            const float * val = vec + BLOCK + 2 * pair;
            float2 v[4];
#pragma unroll
            for (int t = 0; t < 4; t++) v[t] = *reinterpret_cast<const float2 *>(val + t * kCols);
            if (AHEAD) {
                read_update(vec);
                if (c + 1 < n_blocks) read_dots(piece(c + 1));
            }
            float a[16];
#pragma unroll
            for (int v = 0; v < 16; v++) a[v] = dr_both(acc[v >> 3][v & 7]);
            // sixteen sums over the sixteen lanes: the values a lane carries are halved with every exchange; lane l ends with sum l: p_0 ..
            // p_3, r_0 .. r_3 of the first column, then of the second
#pragma unroll
            for (int half = 8; half >= 1; half >>= 1) {
                const bool up = lane & half;
#pragma unroll
                for (int i = 0; i < half; i++) {
                    const float give = up ? a[i] : a[i + half], keep = up ? a[i + half] : a[i];
                    a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * half);
                }
            }
            float u[2][4];
#pragma unroll
            for (int x = 0; x < 2; x++) {
                float p[4];
#pragma unroll
                for (int t = 0; t < 4; t++) p[t] = (x ? v[t].y : v[t].x) - __shfl_sync(0xffffffffu, a[0], 2 * (8 * x + t) + (tid & 1));
                u[x][0] = be.x * p[0];
                u[x][1] = be.y * (p[1] - A0.x * u[x][0]);
                u[x][2] = be.z * (p[2] - (A0.y * u[x][0] + A0.z * u[x][1]));
                u[x][3] = be.w * (p[3] - (A0.w * u[x][0] + A1.x * u[x][1] + A1.y * u[x][2]));
            }
#pragma unroll
            for (int i = 0; i < E / 4; i++) {
                ulonglong2 e = AHEAD ? uv[i][4] : at(vec, 12, i);
#pragma unroll
                for (int x = 0; x < 2; x++) { S[x][2 * i] = mul2(e.x, S[x][2 * i]); S[x][2 * i + 1] = mul2(e.y, S[x][2 * i + 1]); }
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    e = AHEAD ? uv[i][t] : at(vec, 8 + t, i);
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        const unsigned long long w = pack2(u[x][t], u[x][t]);
                        S[x][2 * i] = fma2(e.x, w, S[x][2 * i]);
                        S[x][2 * i + 1] = fma2(e.y, w, S[x][2 * i + 1]);
                    }
                }
            }
            // EVERY: every lane's sum, so that only the store is under a condition.  The other half of the lanes' sums cost more than they save
            // where many CTAs share the units: 100 portions of 40 tokens, 32 heads with a decay a channel 1,648 -> 1,621 us through the mixer without
            // them; 16 heads with a decay a head 578 -> 554 with them
            const int t = 4 * c + (lane & 7) - 4;
            const bool second = lane & 8, mine = (lane & 4) && t < t1 - t0;
            if (EVERY || mine) {
                if (!EVERY) B = *reinterpret_cast<const float4 *>(num + 12 + 4 * (lane & 3));
                const float u0 = second ? u[1][0] : u[0][0], u1 = second ? u[1][1] : u[0][1], u2 = second ? u[1][2] : u[0][2];
                const float u3 = second ? u[1][3] : u[0][3];
                const float o = a[0] + (B.x * u0 + B.y * u1 + B.z * u2 + B.w * u3);
                if (mine) to_out[(long long) t * HV] = o;
            }
        }
    }
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
        for (int i = 0; i < E / 4; i++) {
            ulonglong2 e;
            e.x = S[x][2 * i]; e.y = S[x][2 * i + 1];
            *reinterpret_cast<ulonglong2 *>(scol + x * D + 4 * lane + 4 * kPairLanes * i) = e;
        }
}

}  // namespace iian

using namespace iian;

// Floats of one four-token piece (all heads) of iian_delta_block_scan's scratch.
IIAN_API long long iian_delta_block_floats(int H, int D) { return (long long) H * (13 * D + kBlockNumbers); }

// The scan of iian_delta_scan for bfloat16 models, portions of at_least tokens and more four tokens at a time.  blocks: scratch for N / 4 + S
// pieces with `pieces` 0, else for S * pieces: the step is then walked in segments of 4 * pieces tokens of every sequence, max_q_len the
// most tokens a sequence has.  D 64 or 128, V a multiple of 16.
IIAN_API int iian_delta_block_scan(const float * qn, const float * kn, const float * vv, const float * beta, const float * decay,
                                   const float * qk, float * blocks, int pieces, float * state, long long state_stride, const void * proj, long long ld,
                                   int col_off, int n_taps, const int * cu_q, const int * state_slots, float * out, int N, int S, int H,
                                   int G, int D, int V, int max_q_len, int at_least, int per_head, cudaStream_t stream) {
    if (N <= 0 || S <= 0 || max_q_len <= 0) return IIAN_OK;
    if (H <= 0 || G <= 0 || H % G || (D != 64 && D != 128) || V <= 0 || V % kCols || n_taps < 1 || n_taps > kMaxTaps || pieces < 0 || S > 65535 ||
        H > 65535) return IIAN_ERR_SHAPE;
    if (state_stride % 4 || (((uintptr_t) blocks | (uintptr_t) qn | (uintptr_t) kn | (uintptr_t) vv | (uintptr_t) decay | (uintptr_t) state) & 15))
        return IIAN_ERR_ALIGN;
    typedef __nv_bfloat16 bf;
    const bool ahead = (long long) (V / kCols) * H * S <= 148;
    const int per = max_q_len < 4 * S ? 1 : 2;
    const size_t smem = (size_t) kBlockStages * (ahead ? 2 : per) * (13 * D + kBlockNumbers + 4 * kCols) * sizeof(float);
    auto by_head = [&](auto depth, auto each, auto first) {
        constexpr int E = decltype(depth)::value, PER = decltype(each)::value;
        constexpr bool AHEAD = decltype(first)::value;
        return per_head ? delta_block_scan_kernel<E, PER, AHEAD, true, bf> : delta_block_scan_kernel<E, PER, AHEAD, false, bf>;
    };
    auto by_depth = [&](auto each, auto first) {
        return D == 128 ? by_head(std::integral_constant<int, 8>(), each, first) : by_head(std::integral_constant<int, 4>(), each, first);
    };
    auto scan = ahead ? by_depth(std::integral_constant<int, 2>(), std::true_type())
              : per == 2 ? by_depth(std::integral_constant<int, 2>(), std::false_type()) : by_depth(std::integral_constant<int, 1>(), std::false_type());
    const unsigned threads = kCols / 2 * kPairLanes + (ahead ? 32 : 0);
    const cudaError_t e = cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess) return 1000 + (int) e;
    const int step = pieces > 0 ? 4 * pieces : max_q_len;
    for (int from = 0; from < max_q_len; from += step) {
        const dim3 grid = pieces > 0 ? dim3(min(pieces, (max_q_len - from + 3) / 4), H, S) : dim3(N / 4 + S, H);
        delta_block_kernel<<<grid, 128, 0, stream>>>(qn, kn, beta, decay, per_head, cu_q, state_slots, blocks, from, pieces, at_least, S, H, G, D);
        int rc = iian_launch_status();
        if (rc != IIAN_OK) return rc;
        scan<<<dim3(V / kCols, H, S), threads, smem, stream>>>(blocks, qn, kn, vv, beta, decay, qk, state, state_stride, (long long) H * V * D,
                                                                      (const bf *) proj, ld, col_off, n_taps, cu_q, state_slots, out, from, pieces,
                                                                      at_least, H, G, V);
        rc = iian_launch_status();
        if (rc != IIAN_OK) return rc;
    }
    return IIAN_OK;
}

// Floats of a slot's state: S [H, V, D], then the tail [taps - 1, 2 G D + H V].
IIAN_API long long iian_delta_state_floats(int H, int G, int D, int V, int n_taps) {
    return (long long) H * V * D + (long long) (n_taps - 1) * (2LL * G * D + (long long) H * V);
}

template <bool HEAD, typename A>
static int launch_prep(const A * proj, long long ld, int col_off, int b_off, const float * b_pre, const float * z, long long ld_z,
                       const float * taps, int n_taps, const float * a_log, const float * dt_bias, const float * state,
                       long long state_stride, const int * seq_of_token, const int * cu_q, const int * state_slots, float * qn,
                       float * kn, float * vv, float * beta, float * decay, float * qk, int N, int H, int G, int D, int V,
                       cudaStream_t stream) {
    const long long tail_off = (long long) H * V * D;
    const float q_scale = 1.0f / sqrtf((float) D);
    if constexpr (std::is_same<A, __nv_bfloat16>::value) {
        const bool whole = ld % 4 == 0 && col_off % 4 == 0 && ((uintptr_t) proj & 7) == 0 && (HEAD || (ld_z % 4 == 0 && ((uintptr_t) z & 15) == 0)) &&
                           (((uintptr_t) taps | (uintptr_t) dt_bias | (uintptr_t) qn | (uintptr_t) kn | (uintptr_t) vv | (uintptr_t) decay) & 15) == 0;
        if (N >= kPrepTileFrom && D == 128 && V % 128 == 0 && n_taps == 4 && whole) {
            const int units = G + H * V / 128 + H;
            // rows a warp walks: the more the fewer windows are begun, but the grid should be two rounds of CTAs (three an SM): 16 heads with a
            // decay per channel, 4, 8 and 16 rows: 256 tokens 8.6, 13.4, 23.2 us (tiles 13.8), 768 20.5, 19.3, 25.1 (29.7), 1,500 37.3, 35.5,
            // 34.8 (54.2)
            auto ctas = [&](int T) { return (long long) ((N + T - 1) / T) * ((units + kWideWarps - 1) / kWideWarps); };
            auto go = [&](auto tokens) {
                constexpr int T = decltype(tokens)::value;
                return iian_launch(delta_prep_wide_kernel<HEAD, T>, dim3((N + T - 1) / T, (units + kWideWarps - 1) / kWideWarps),
                                   dim3(kWideWarps * 32), 0, stream, proj, ld, col_off, b_off, b_pre, z, ld_z, taps, a_log, dt_bias, state, state_stride,
                                   tail_off, seq_of_token, cu_q, state_slots, qn, kn, vv, beta, decay, qk, N, H, G, V, q_scale);
            };
            if (ctas(16) >= 6 * 148) return go(std::integral_constant<int, 16>());
            return ctas(8) >= 6 * 148 ? go(std::integral_constant<int, 8>()) : go(std::integral_constant<int, 4>());
        }
    }
    // many tokens: tiles of T rows through shared memory; few: a CTA per token and unit, so that they spread over the GPU
    int T = N >= 4 * kPrepTileFrom ? 16 : N >= kPrepTileFrom ? 8 : 0;
    size_t smem = 0;
    const int W = 2 * D > V ? 2 * D : V;
    for (; T >= 4; T /= 2) {
        smem = ((size_t) (T + n_taps - 1) * W + (size_t) W * n_taps + 2 * T) * sizeof(float);
        if (smem <= 96 * 1024) break;
    }
    if (T >= 4) {
        const dim3 tgrid((N + T - 1) / T, G + H);
        if (smem > 48 * 1024) cudaFuncSetAttribute(delta_prep_tile_kernel<HEAD, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        return iian_launch(delta_prep_tile_kernel<HEAD, A>, tgrid, dim3(kPrepTileWarps * 32), smem, stream, proj, ld, col_off, b_off, b_pre,
                           z, ld_z, taps, n_taps, a_log, dt_bias, state, state_stride, tail_off, seq_of_token, cu_q, state_slots, qn, kn,
                           vv, beta, decay, qk, N, T, H, G, D, V, q_scale);
    }
    return iian_launch(delta_prep_kernel<HEAD, A>, dim3(N, G + H), dim3(kPrepThreads), 0, stream, proj, ld, col_off, b_off, b_pre, z, ld_z,
                       taps, n_taps, a_log, dt_bias, state, state_stride, tail_off, seq_of_token, cu_q, state_slots, qn, kn, vv, beta,
                       decay, qk, H, G, D, V, q_scale);
}

// per_head: one decay per head (z, dt_bias and decay hold H numbers per token) instead of one per key channel (H * D).
// b_pre: float32 pre-activations of the write strengths (row stride ld_z), or null: the columns of proj at b_off.
IIAN_API int iian_delta_prep(const void * proj, long long ld, int col_off, int b_off, int act_dtype, const float * b_pre, const float * z,
                             long long ld_z, int per_head, const float * taps, int n_taps, const float * a_log, const float * dt_bias,
                             const float * state, long long state_stride, const int * seq_of_token, const int * cu_q,
                             const int * state_slots, float * qn, float * kn, float * vv, float * beta, float * decay, float * qk,
                             int N, int H, int G, int D, int V, cudaStream_t stream) {
    if (N <= 0) return IIAN_OK;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || V <= 0 || n_taps < 1 || n_taps > kMaxTaps) return IIAN_ERR_SHAPE;
    if (D > kPrepMaxDim) return IIAN_ERR_LIMIT;
    if (G + H > 65535) return IIAN_ERR_LIMIT;
#define IIAN_PREP(HEAD, A) return launch_prep<HEAD, A>((const A *) proj, ld, col_off, b_off, b_pre, z, ld_z, taps, n_taps, a_log, dt_bias, \
                                                       state, state_stride, seq_of_token, cu_q, state_slots, qn, kn, vv, beta, decay, qk, \
                                                       N, H, G, D, V, stream)
    if (act_dtype == IIAN_F32) { if (per_head) IIAN_PREP(true, float); IIAN_PREP(false, float); }
    if (act_dtype == IIAN_BF16) { if (per_head) IIAN_PREP(true, __nv_bfloat16); IIAN_PREP(false, __nv_bfloat16); }
#undef IIAN_PREP
    return IIAN_ERR_DTYPE;
}

template <int E, bool HEAD, typename A>
static int launch_scan(const float * qn, const float * kn, const float * vv, const float * beta, const float * decay,
                       const float * qk, float * state, long long state_stride, const A * proj, long long ld, int col_off,
                       int n_taps, const int * cu_q, const int * state_slots, float * out, int S, int H, int G, int D, int V,
                       int max_q_len, bool vec, cudaStream_t stream) {
    const int Dp = (D + 3) & ~3;
    int chunk = D <= 256 ? 16 : 8;             // tokens per stage of shared memory
    if (max_q_len > 0 && max_q_len < chunk) chunk = max_q_len;         // single tokens: small stages, more CTAs per SM
    const size_t smem = (size_t) scan_floats(HEAD, Dp, chunk) * sizeof(float);
    if (smem > 200 * 1024) return IIAN_ERR_LIMIT;
    const dim3 grid((V + kCols - 1) / kCols, H, S);
    if constexpr (E % 4 == 0) if (vec) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(delta_scan_kernel<E, true, HEAD, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        return iian_launch(delta_scan_kernel<E, true, HEAD, A>, grid, dim3(kCols * kLanes), smem, stream, qn, kn, vv, beta, decay, qk, state,
                           state_stride, (long long) H * V * D, proj, ld, col_off, n_taps, cu_q, state_slots, out, H, G, D, V, chunk);
    }
    if (smem > 48 * 1024) cudaFuncSetAttribute(delta_scan_kernel<E, false, HEAD, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    return iian_launch(delta_scan_kernel<E, false, HEAD, A>, grid, dim3(kCols * kLanes), smem, stream, qn, kn, vv, beta, decay, qk, state,
                       state_stride, (long long) H * V * D, proj, ld, col_off, n_taps, cu_q, state_slots, out, H, G, D, V, chunk);
}

template <bool HEAD, typename A>
static int scan_by_depth(const float * qn, const float * kn, const float * vv, const float * beta, const float * decay,
                         const float * qk, float * state, long long state_stride, const A * proj, long long ld, int col_off,
                         int n_taps, const int * cu_q, const int * state_slots, float * out, int S, int H, int G, int D, int V,
                         int max_q_len, cudaStream_t stream) {
    const int e = (D + kLanes - 1) / kLanes;
    const bool vec = D % 4 == 0 && state_stride % 4 == 0 &&
                     (((uintptr_t) qn | (uintptr_t) kn | (uintptr_t) decay | (uintptr_t) state) & 15) == 0;
#define IIAN_SCAN(E) return launch_scan<E, HEAD, A>(qn, kn, vv, beta, decay, qk, state, state_stride, proj, ld, col_off, n_taps, cu_q, \
                                              state_slots, out, S, H, G, D, V, max_q_len, vec, stream)
    if (e <= 2 && !vec) IIAN_SCAN(2);
    if (e <= 4) IIAN_SCAN(4);
    if (e <= 8) IIAN_SCAN(8);
    if (e <= 16) IIAN_SCAN(16);
    if (e <= 32) IIAN_SCAN(32);
    if (e <= 64) IIAN_SCAN(64);
#undef IIAN_SCAN
    return IIAN_ERR_LIMIT;
}

// out: float32 [N, H * V].  per_head: decay is [N, H] instead of [N, H * D].  S sequences (grid z); a sequence with state slot -1 is padding.  max_q_len: the most tokens a
// sequence has in this step (0: unknown); it sizes the stages of shared memory.
IIAN_API int iian_delta_scan(const float * qn, const float * kn, const float * vv, const float * beta, const float * decay,
                             const float * qk, float * state, long long state_stride, const void * proj, long long ld,
                             int col_off, int act_dtype, int n_taps, const int * cu_q, const int * state_slots, float * out,
                             int S, int H, int G, int D, int V, int max_q_len, int per_head,
                            cudaStream_t stream) {
    if (S <= 0) return IIAN_OK;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || V <= 0 || n_taps < 1 || n_taps > kMaxTaps || S > 65535 || H > 65535) return IIAN_ERR_SHAPE;
#define IIAN_SCAN_AS(HEAD, A) return scan_by_depth<HEAD, A>(qn, kn, vv, beta, decay, qk, state, state_stride, (const A *) proj, ld, col_off, \
                                                            n_taps, cu_q, state_slots, out, S, H, G, D, V, max_q_len, stream)
    if (act_dtype == IIAN_F32) { if (per_head) IIAN_SCAN_AS(true, float); IIAN_SCAN_AS(false, float); }
    if (act_dtype == IIAN_BF16) { if (per_head) IIAN_SCAN_AS(true, __nv_bfloat16); IIAN_SCAN_AS(false, __nv_bfloat16); }
#undef IIAN_SCAN_AS
    return IIAN_ERR_DTYPE;
}
