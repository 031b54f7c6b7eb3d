// layout.cuh -- layout passes between the MEX-native cell-major arrays and the tiled
// cell-fastest layout the contraction kernels read (see common.cuh).  Included by plan.cu only.
#pragma once
#include "common.cuh"

namespace cf {

// ----------------------------------------------------------------------------------------
// Layout passes: MEX-native cell-major [B][N_Q*K] (m = q + k*N_Q)  <->  tiled [tile][q*K+k][32]
// ----------------------------------------------------------------------------------------
template <typename TO>
__global__ void __launch_bounds__(256) pack_tiles_kernel(const double* __restrict__ src,
                                                         TO* __restrict__ dst, int64_t B,
                                                         int nq, int K) {
    __shared__ double sm[32][33];
    const int M = nq * K;
    const int64_t tile = blockIdx.y;
    const int m0 = blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int c = ty; c < 32; c += 8) {
        const int64_t b = tile * 32 + c;
        const int m = m0 + tx;
        sm[c][tx] = (b < B && m < M) ? src[b * M + m] : 0.0;
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        const int m = m0 + j;
        if (m < M) {
            const int q = m % nq, k = m / nq;
            dst[(tile * M + (int64_t)q * K + k) * 32 + tx] = (TO)sm[tx][j];
        }
    }
}

static __global__ void __launch_bounds__(256) unpack_tiles_kernel(const double* __restrict__ src,
                                                           double* __restrict__ dst, int64_t B,
                                                           int nq, int K) {
    __shared__ double sm[32][33];
    const int M = nq * K;
    const int64_t tile = blockIdx.y;
    const int m0 = blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int j = ty; j < 32; j += 8) {
        const int m = m0 + j;
        double v = 0.0;
        if (m < M) {
            const int q = m % nq, k = m / nq;
            v = src[(tile * M + (int64_t)q * K + k) * 32 + tx];
        }
        sm[j][tx] = v;
    }
    __syncthreads();
    for (int c = ty; c < 32; c += 8) {
        const int64_t b = tile * 32 + c;
        const int m = m0 + tx;
        if (b < B && m < M) dst[b * M + m] = sm[tx][c];
    }
}

// R in FP32; at K = 8 (RT not null) also R_t as [k1][8 k2 + k3], and that split into BF16 hi + lo (each rounded to
// nearest even), [t][hi, lo][k1][8 k2 + k3].
__device__ __forceinline__ unsigned short bf16_round(float x) {
    uint32_t u = __float_as_uint(x);
    u += 0x7fffu + ((u >> 16) & 1u);
    return (unsigned short)(u >> 16);
}
static __global__ void __launch_bounds__(256) derive_r_kernel(const double* __restrict__ R, float* __restrict__ R32,
                                                              double* __restrict__ RT, unsigned short* __restrict__ RTbf,
                                                              size_t n) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const double r = R[i];
    R32[i] = (float)r;
    if (RT == nullptr) return;
    const size_t t = i / 512;
    const int e = (int)(i % 512), j = (e % 8) * 64 + (e / 8) % 8 * 8 + e / 64;
    RT[t * 512 + j] = r;
    const unsigned short hi = bf16_round((float)r);
    RTbf[t * 1024 + j] = hi;
    RTbf[t * 1024 + 512 + j] = bf16_round((float)(r - (double)__uint_as_float((uint32_t)hi << 16)));
}

// R_t in the lane order of the outer-product kernels: dst[(t K + k1) 32 + lane] = R_t[k1][k2 = lane / 4][k3 = 2 (lane % 4),
// + 1], zero where k2 or k3 is past K.
static __global__ void __launch_bounds__(256) lane_order_kernel(const double* __restrict__ R, double2* __restrict__ dst,
                                                                size_t n, int K) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int lane = (int)(i % 32), k2 = lane >> 2, k3 = 2 * (lane & 3);
    const size_t tk = i / 32, t = tk / K, k1 = tk % K;
    const double* src = R + t * K * K * K + k1 + (size_t)K * k2 + (size_t)K * K * k3;
    dst[i] = make_double2(k2 < K && k3 < K ? src[0] : 0.0, k2 < K && k3 + 1 < K ? src[(size_t)K * K] : 0.0);
}

// FP64 FMA throughput probe: kProbeChains independent DFMA chains per thread.
constexpr int kProbeChains = 8;
static __global__ void __launch_bounds__(256) fp64_fma_probe_kernel(double* sink, int iters, double a) {
    double x[kProbeChains];
#pragma unroll
    for (int c = 0; c < kProbeChains; ++c) x[c] = threadIdx.x * 1e-3 + c;
    const double b = 1e-9;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int c = 0; c < kProbeChains; ++c) x[c] = fma(x[c], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < kProbeChains; ++c) s += x[c];
    sink[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace cf
