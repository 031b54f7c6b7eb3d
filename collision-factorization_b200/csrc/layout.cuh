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

// Chunks of the outer-product kernels (outer_kernels.cuh): four runs of equal q2, each with one or two q3, as byte
// offsets in a row of cell pairs (four words), and their G (eight words).  While it is made, a run is three words, q2 | q3a
// << 16 | q3b << 32 | two << 48 and its two G, so that four runs lie where their chunk will.
constexpr int kOuterChunkWords = 12;
struct OuterRun {
    unsigned long long q;
    double ga, gb;
    __device__ int q2() const { return (int)(q & 0xffff); }
    __device__ int qa() const { return (int)(q >> 16 & 0xffff); }
    __device__ int qb() const { return (int)(q >> 32 & 0xffff); }
    __device__ bool two() const { return q >> 48; }
};
__device__ __forceinline__ unsigned long long outer_word(int q2, int qa, int qb, int two) {
    return (unsigned long long)q2 | (unsigned long long)qa << 16 | (unsigned long long)qb << 32 | (unsigned long long)two << 48;
}

// A thread per slice: the slice's entries as runs in the order of q2, the runs of two in front, then four runs to a chunk.
// The runs of a chunk are picked so that their q2, and their q3 of either column, are distinct modulo 4 as far as a
// few candidates allow (the operands of eight lanes then lie in distinct banks: 20 % above the conflict-free count at
// L = 10, 39 % in the list's own order).  The runs lie where their chunks will, four in the place of one; empty
// places read one of the n_zero rows of zeros behind the last q.
static __global__ void __launch_bounds__(64) pack_chunks_kernel(const int* __restrict__ slice_e, const uint32_t* __restrict__ e_q23,
                                                                const double* __restrict__ e_g, const int4* __restrict__ place,
                                                                int n_slices, int n_q, int n_zero, unsigned long long* chunks) {
    constexpr int kLook = 6;  // candidates per place
    const int s = blockIdx.x * 64 + threadIdx.x;
    if (s >= n_slices) return;
    const int4 pl = place[s];
    const int e0 = slice_e[s], e1 = slice_e[s + 1], n_two = pl.y, n_all = pl.z;
    unsigned long long* w = chunks + (size_t)pl.x * kOuterChunkWords;
    auto get = [&](int i) { return OuterRun{w[3 * i], __longlong_as_double(w[3 * i + 1]), __longlong_as_double(w[3 * i + 2])}; };
    auto put = [&](int i, const OuterRun& r) {
        w[3 * i] = r.q;
        w[3 * i + 1] = __double_as_longlong(r.ga);
        w[3 * i + 2] = __double_as_longlong(r.gb);
    };
    int i_two = 0, i_one = n_two;
    for (int q2 = -1;;) {
        int next = 0x10000, first = e0;
        for (int e = e0; e < e1; ++e) {
            const int q = e_q23[e] & 0xffffu;
            if (q > q2 && q < next) {
                next = q;
                first = e;
            }
        }
        if (next == 0x10000) break;
        q2 = next;
        int held = -1;  // an entry that waits for its second
        for (int e = first; e < e1; ++e) {
            if ((int)(e_q23[e] & 0xffffu) != q2) continue;
            if (held < 0) {
                held = e;
                continue;
            }
            put(i_two++, {outer_word(q2, e_q23[held] >> 16, e_q23[e] >> 16, 1), e_g[held], e_g[e]});
            held = -1;
        }
        if (held >= 0) {
            const int q3 = e_q23[held] >> 16;
            put(i_one++, {outer_word(q2, q3, q3, 0), e_g[held], 0.0});
        }
    }
    for (int i0 = 0; i0 < n_all; i0 += 4) {
        uint32_t used[3] = {};  // runs of this chunk per residue (a byte each): q2, q3a, q3b
        auto in = [&](int kind, int q) { return (int)(used[kind] >> 8 * (q & 3) & 0xffu); };
        auto take = [&](int kind, int q) { used[kind] += 1u << 8 * (q & 3); };
        for (int i = i0; i < min(i0 + 4, n_all); ++i) {
            const int hi = min(i + kLook, i < n_two ? n_two : n_all);  // runs of two stay in front
            int best = i, c_best = 1 << 20;
            bool flip = false;
            for (int c = i; c < hi && c_best > 0; ++c) {
                const OuterRun r = get(c);
                const int c2 = in(0, r.q2()), a0 = in(1, r.qa()) + in(2, r.qb()), a1 = in(1, r.qb()) + in(2, r.qa());
                if (c2 + min(a0, a1) < c_best) {
                    c_best = c2 + min(a0, a1);
                    best = c;
                    flip = r.two() && a1 < a0;
                }
            }
            OuterRun r = get(best);
            if (best != i) put(best, get(i));
            if (flip) r = {outer_word(r.q2(), r.qb(), r.qa(), 1), r.gb, r.ga};
            put(i, r);
            take(0, r.q2());
            take(1, r.qa());
            take(2, r.qb());
        }
        // the row of zeros in the residue that the fewest others of its kind have
        auto zero_row = [&](int kind) {
            int best = n_q;
            for (int q = n_q + 1; q < n_q + n_zero; ++q)
                if (in(kind, q) < in(kind, best)) best = q;
            take(kind, best);
            return best;
        };
        const bool two = i0 < n_two;  // the kernel reads q3b too
        OuterRun r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            r[i] = i0 + i < n_all ? get(i0 + i) : OuterRun{0, 0.0, 0.0};
            const int q2 = i0 + i < n_all ? r[i].q2() : zero_row(0), qa = i0 + i < n_all ? r[i].qa() : zero_row(1),
                      qb = i0 + i < n_all && (r[i].two() || !two) ? r[i].qb() : zero_row(2);
            r[i].q = outer_word(16 * q2, 16 * qa, 16 * qb, 0);
        }
        unsigned long long* ch = w + i0 / 4 * kOuterChunkWords;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ch[i] = r[i].q;
            ch[4 + 2 * i] = __double_as_longlong(r[i].ga);
            ch[5 + 2 * i] = __double_as_longlong(r[i].gb);
        }
    }
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
