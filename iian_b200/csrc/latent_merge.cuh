// The parts of a row's keys put together: what the two tensor-core kernels of the attention over a cached latent share.
#pragma once
#include "common.cuh"

namespace iian {

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned *>(&v);
}

// out[row] = sum_z o_z exp(m_z - m) / sum_z l_z exp(m_z - m),  z ascending
static __global__ void latent_merge_kernel(const float * __restrict__ part_o, const float * __restrict__ part_ml,
                                    __nv_bfloat16 * __restrict__ out, const int * __restrict__ seq_of_token, int H, int parts,
                                    int rank) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float wz[64];                  // the weight of every part: exp(m_z - m) / l
    const size_t row = blockIdx.x;
    if (seq_of_token[row / H] < 0) {
        for (int c = threadIdx.x; c < rank; c += blockDim.x) out[row * rank + c] = __float2bfloat16_rn(0.0f);
        return;
    }
    if (threadIdx.x < 32) {
        const int z = threadIdx.x;
        const float mz = z < parts ? part_ml[(row * parts + z) * 2] : -INFINITY;
        const float lz = z < parts ? part_ml[(row * parts + z) * 2 + 1] : 0.0f;
        const float m = warp_max(mz);
        const float e = mz == -INFINITY ? 0.0f : __expf(mz - m);
        float l = lz * e;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {     // in the order of the parts: a prefix-style sum keeps z ascending pairs together
            l += __shfl_xor_sync(0xffffffffu, l, o);
        }
        wz[z] = l > 0.0f ? e / l : 0.0f;
    }
    __syncthreads();
    const float * po = part_o + row * parts * rank;
    for (int c = threadIdx.x * 2; c < rank; c += blockDim.x * 2) {
        float a0 = 0.0f, a1 = 0.0f;
        for (int z = 0; z < parts; z++) {
            const float2 v = *reinterpret_cast<const float2 *>(po + (size_t) z * rank + c);
            a0 = fmaf(v.x, wz[z], a0);
            a1 = fmaf(v.y, wz[z], a1);
        }
        *reinterpret_cast<unsigned *>(out + row * rank + c) = pack_bf16(a0, a1);
    }
}

static inline int latent_merge(const float * part_o, const float * part_ml, void * out, const int * seq_of_token, int N, int H, int parts,
                               int rank, cudaStream_t stream) {
    return iian_launch(latent_merge_kernel, dim3((unsigned) ((size_t) N * H)), dim3(rank >= 256 ? 128 : 64), 0, stream, part_o, part_ml,
                       (__nv_bfloat16 *) out, seq_of_token, H, parts, rank);
}

}  // namespace iian
