// krylov.cu -- batched implicit solves (I - dt J(f)) x = b with restarted GMRES, FP64, on the GPU.
//
// Every cell has its own f, hence its own Jacobian, and its own Krylov space.  All vectors live in
// the tiled cell layout [ceil(B/32)][N_Q*K][32] (lane = cell), so every vector kernel below is a
// coalesced stream with one cell per lane, and a matrix-vector product is one batched J.v launch
// of the contraction library (cf_jv_tiled) plus an axpy.
//
//   * right preconditioning: A P^-1 u = b, x = P^-1 u, so the Arnoldi residual is the true one;
//   * P^-1 is block-Jacobi over the angular modes q: N_Q blocks of K x K, either shared by all
//     cells (the Maxwellian-linearised blocks of I - dt J_eq, tutorial_chapman_enscog_decay_rates.m:42-48
//     generalised) or one set per cell (the learned preconditioner);
//   * classical Gram-Schmidt with one re-orthogonalisation (CGS2), FP64;
//   * Givens rotations per cell; a cell stops extending its Krylov space once its estimated residual
//     reaches tol * |b|, and the restart's true residual b - A x is recomputed in FP64.
//
// The host drives the iteration.  An Arnoldi step is the J.v launch and one k_step launch, in which a CTA does all of
// a 16-cell half-tile's vector work: its vectors are 128-byte rows that no other CTA touches, so both
// Gram-Schmidt sweeps, the Givens rotation, the new basis vector and its preconditioned image need no
// grid-wide step between them, and the basis is read three times (h; w' = w - V h with V^T w' in the same
// pass; w'' = w' - V hh) instead of four.  Cells converge at different steps; once a quarter of them are
// done, J.v runs on the active cells gathered into whole tiles.
// B200, L = 8, K = 8, 2048 cells, dt nu = 10, block preconditioner: 8.0 ms a solve, 6.4 of them J.v and 1.0 k_step;
// 16.8 ms with one launch per vector operation on 64 CTAs (k_dots alone 5.6 ms) and J.v of every cell until the
// last had converged (8 to 14 steps).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/cf_b200.h"

void cf_set_last_error(const char* msg);

namespace {

constexpr int kLanes = 32;
constexpr int kHalf = 16;           // cells per CTA of the vector kernels
constexpr int kVecThreads = 512;
constexpr int kVecWarps = kVecThreads / 32;
constexpr int kRowGroups = kVecThreads / kHalf;  // rows in flight: thread (c = tid % 16, rg = tid / 16)
constexpr int kMaxBasis = 64;       // restart <= 63
constexpr int kMaxK = 16;

// Per-cell state of the Arnoldi process.
struct CellState {
    double* H;        // [m+1][m][cells]   H[i][j] at (i*m + j)*cells + c
    double* cs;       // [m][cells]
    double* sn;       // [m][cells]
    double* g;        // [m+1][cells]
    double* bnorm;    // [cells]
    int* kdim;        // [cells] Krylov dimension in use (frozen cells keep theirs)
    int* active;      // [cells]
};


// What every vector kernel needs: the tiled layout of one half-tile and the preconditioner.
struct Geo {
    int nq, K, M, n_cells;
    size_t C, vec;  // padded cells, doubles per vector
    const double* P;
    int per_cell;
};

// out[i][c] = sum over the CTA's threads of acc[i] for its cell c, i < n (in a fixed order).
template <int NV>
__device__ __forceinline__ void reduce_cells(const double (&acc)[NV], int n, double* out, double (*red)[8][kHalf]) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int i0 = 0; i0 < NV; i0 += 8) {
        if (i0 >= n) break;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const double x = i0 + k < NV ? acc[i0 + k < NV ? i0 + k : 0] : 0.0;
            const double a = x + __shfl_xor_sync(0xffffffffu, x, 16);
            if (lane < kHalf) red[warp][k][lane] = a;
        }
        __syncthreads();
        if (tid < 8 * kHalf && i0 + tid / kHalf < n) {
            double s = 0.0;
            for (int w = 0; w < kVecWarps; ++w) s += red[w][tid / kHalf][tid % kHalf];
            out[(i0 + tid / kHalf) * kHalf + tid % kHalf] = s;
        }
        __syncthreads();
    }
}

// z = P v for the half-tile's cells, v = the row values that value(row) gives for this thread's cell; put(row, v)
// is called with each of them.
template <typename Value, typename Put>
__device__ __forceinline__ void precondition(const Geo& g, size_t base, size_t cell, double* __restrict__ z, Value value,
                                             Put put) {
    const int rg = threadIdx.x / kHalf;
    for (int q = rg; q < g.nq; q += kRowGroups) {
        double v[kMaxK];
#pragma unroll
        for (int b = 0; b < kMaxK; ++b)
            if (b < g.K) {
                v[b] = value(q * g.K + b);
                put(q * g.K + b, v[b]);
            }
        const double* Pq =
            g.P ? g.P + ((g.per_cell ? (cell < (size_t)g.n_cells ? cell : 0) * (size_t)g.nq : 0) + q) * (size_t)g.K * g.K
                : nullptr;
#pragma unroll
        for (int a = 0; a < kMaxK; ++a)
            if (a < g.K) {
                double s = 0.0;
                if (Pq) {
#pragma unroll
                    for (int b = 0; b < kMaxK; ++b)
                        if (b < g.K) s = fma(__ldg(Pq + a * g.K + b), v[b], s);
                } else {
                    s = v[a];
                }
                z[base + (size_t)(q * g.K + a) * kLanes] = s;
            }
    }
}

// |b| per cell.
__global__ void __launch_bounds__(kVecThreads) k_bnorm(Geo g, const double* __restrict__ b, double* __restrict__ bnorm) {
    __shared__ double red[kVecWarps][8][kHalf], sum[kHalf];
    const int tid = threadIdx.x, c = tid % kHalf, rg = tid / kHalf;
    const size_t cell = (size_t)blockIdx.x * kHalf + c;
    const size_t base = cell / kLanes * g.M * kLanes + cell % kLanes;
    double acc[1] = {0.0};
    for (int r = rg; r < g.M; r += kRowGroups) {
        const double x = b[base + (size_t)r * kLanes];
        acc[0] = fma(x, x, acc[0]);
    }
    reduce_cells<1>(acc, 1, sum, red);
    if (tid < kHalf) bnorm[(size_t)blockIdx.x * kHalf + tid] = sqrt(fmax(sum[tid], 0.0));
}

// True residual r = b - (x - dt J x) and the start of a cycle: relative residuals, cells above tol counted and made
// active, V0 = r / |r|, z = P V0.  jx holds J x.
__global__ void __launch_bounds__(kVecThreads)
    k_residual(Geo g, CellState st, const double* __restrict__ b, const double* __restrict__ x,
               const double* __restrict__ jx, double* __restrict__ r, double* __restrict__ V0, double* __restrict__ z,
               double dt, double* __restrict__ rel, int* __restrict__ n_bad, int m, double tol) {
    __shared__ double red[kVecWarps][8][kHalf], sum[kHalf], scale[kHalf];
    const int tid = threadIdx.x, c = tid % kHalf, rg = tid / kHalf;
    const size_t cell = (size_t)blockIdx.x * kHalf + c;
    const size_t base = cell / kLanes * g.M * kLanes + cell % kLanes;
    double acc[1] = {0.0};
    for (int row = rg; row < g.M; row += kRowGroups) {
        const size_t i = base + (size_t)row * kLanes;
        const double v = b[i] - (x[i] - dt * jx[i]);
        r[i] = v;
        acc[0] = fma(v, v, acc[0]);
    }
    reduce_cells<1>(acc, 1, sum, red);
    if (tid < kHalf) {
        const size_t cc = (size_t)blockIdx.x * kHalf + tid;
        const double beta = sqrt(fmax(sum[tid], 0.0)), bn = st.bnorm[cc];
        for (int i = 0; i <= m; ++i) st.g[(size_t)i * g.C + cc] = 0.0;
        st.g[cc] = beta;
        st.kdim[cc] = 0;
        const bool act = cc < (size_t)g.n_cells && beta > tol * bn;
        st.active[cc] = act ? 1 : 0;
        scale[tid] = act ? 1.0 / beta : 0.0;
        if (cc < (size_t)g.n_cells) {
            const double v = bn > 0 ? beta / bn : beta;
            rel[cc] = v;
            if (v > tol) atomicAdd(n_bad, 1);
        }
    }
    __syncthreads();
    const double sc = scale[c];
    precondition(g, base, cell, z, [&](int row) { return r[base + (size_t)row * kLanes] * sc; },
                 [&](int row, double v) { V0[base + (size_t)row * kLanes] = v; });
}

// One Arnoldi step for a half-tile: w = z - dt J z orthogonalised twice against V_0..V_j, the Givens rotation,
// V_(j+1) = w / |w| and z = P V_(j+1); cells that are done get zero vectors.  jz is J z of the whole batch, or, with
// pos, of the gathered active cells (pos[cell] is a cell's place there).
// Three reads of the basis, bound by their latency and L2 bandwidth.  NV: the next size at or above that of the
// basis, whose rows a thread loads together, without branches between the loads (vectors past the last
// one repeat it with h = 0), and holds in registers in the second pass; a basis above 16 takes that pass as two.
template <int NV>
__global__ void __launch_bounds__(kVecThreads)
    k_step(Geo g, CellState st, double* __restrict__ V, double* __restrict__ w, double* __restrict__ z,
           const double* __restrict__ jz, const int* __restrict__ pos, double dt, int j, int m, double tol) {
    __shared__ double red[kVecWarps][8][kHalf];
    __shared__ double h[kMaxBasis * kHalf], hh[kMaxBasis * kHalf];
    __shared__ double norm2[kHalf], inv[kHalf];
    __shared__ int any;
    const int tid = threadIdx.x, c = tid % kHalf, rg = tid / kHalf;
    const size_t cell0 = (size_t)blockIdx.x * kHalf, cell = cell0 + c;
    if (tid == 0) any = 0;
    __syncthreads();
    const bool active = st.active[cell];
    if (tid < kHalf && active) any = 1;
    __syncthreads();
    if (!any) return;
    const size_t base = cell / kLanes * g.M * kLanes + cell % kLanes;
    const int nv = j + 1;
    for (int e = tid; e < kMaxBasis * kHalf; e += kVecThreads) h[e] = hh[e] = 0.0;
    size_t jbase = base;
    if (pos) {
        const size_t p = active ? pos[cell] : 0;
        jbase = p / kLanes * g.M * kLanes + p % kLanes;
    }

    auto load = [&](double (&v)[NV], int i0, size_t at) {
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = V[(size_t)min(i0 + i, nv - 1) * g.vec + at];
    };

    // w = z - dt J z, h = V^T w
    for (int i0 = 0; i0 < nv; i0 += NV) {
        double acc[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] = 0.0;
        for (int r = rg; r < g.M; r += kRowGroups) {
            const size_t at = base + (size_t)r * kLanes;
            double x;
            if (i0 == 0) {
                x = active ? z[at] - dt * jz[jbase + (size_t)r * kLanes] : 0.0;
                w[at] = x;
            } else {
                x = w[at];
            }
            double v[NV];
            load(v, i0, at);
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[i] = fma(v[i], x, acc[i]);
        }
        reduce_cells<NV>(acc, min(NV, nv - i0), h + i0 * kHalf, red);
    }
    // w' = w - V h, hh = V^T w'
    if (nv <= NV) {
        double acc[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] = 0.0;
        for (int r = rg; r < g.M; r += kRowGroups) {
            const size_t at = base + (size_t)r * kLanes;
            double v[NV], s = 0.0;
            const double w0 = w[at];
            load(v, 0, at);
#pragma unroll
            for (int i = 0; i < NV; ++i) s = fma(h[i * kHalf + c], v[i], s);
            const double x = w0 - s;
            w[at] = x;
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[i] = fma(v[i], x, acc[i]);
        }
        reduce_cells<NV>(acc, nv, hh, red);
    } else {
        for (int r = rg; r < g.M; r += kRowGroups) {
            const size_t at = base + (size_t)r * kLanes;
            double s = 0.0;
            for (int i0 = 0; i0 < nv; i0 += NV) {
                double v[NV];
                load(v, i0, at);
#pragma unroll
                for (int i = 0; i < NV; ++i) s = fma(h[(i0 + i) * kHalf + c], v[i], s);
            }
            w[at] -= s;
        }
        for (int i0 = 0; i0 < nv; i0 += NV) {
            double acc[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[i] = 0.0;
            for (int r = rg; r < g.M; r += kRowGroups) {
                const size_t at = base + (size_t)r * kLanes;
                const double x = w[at];
                double v[NV];
                load(v, i0, at);
#pragma unroll
                for (int i = 0; i < NV; ++i) acc[i] = fma(v[i], x, acc[i]);
            }
            reduce_cells<NV>(acc, min(NV, nv - i0), hh + i0 * kHalf, red);
        }
    }
    // w'' = w' - V hh and its norm
    {
        double acc[1] = {0.0};
        for (int r = rg; r < g.M; r += kRowGroups) {
            const size_t at = base + (size_t)r * kLanes;
            double s = 0.0;
            const double w0 = w[at];
            for (int i0 = 0; i0 < nv; i0 += NV) {
                double v[NV];
                load(v, i0, at);
#pragma unroll
                for (int i = 0; i < NV; ++i) s = fma(hh[(i0 + i) * kHalf + c], v[i], s);
            }
            const double x = w0 - s;
            w[at] = x;
            acc[0] = fma(x, x, acc[0]);
        }
        reduce_cells<1>(acc, 1, norm2, red);
    }
    // the column of H through the previous rotations (staged where the reductions are done with), the new
    // rotation, the residual estimate
    double* csn = &red[0][0][0];  // [2][j <= 63][cells]
    static_assert(sizeof(red) >= 2 * (kMaxBasis - 1) * kHalf * sizeof(double), "rotations fit");
    for (int e = tid; e < j * kHalf; e += kVecThreads) {
        const size_t at = (size_t)(e / kHalf) * g.C + cell0 + e % kHalf;
        csn[e] = st.cs[at];
        csn[j * kHalf + e] = st.sn[at];
    }
    __syncthreads();
    if (tid < kHalf) {
        const size_t C = g.C, cc = cell0 + tid;
        inv[tid] = 0.0;
        if (active) {
            const double hn = sqrt(fmax(norm2[tid], 0.0));
            double a = h[tid] + hh[tid];
            for (int i = 0; i < j; ++i) {
                const double b = h[(i + 1) * kHalf + tid] + hh[(i + 1) * kHalf + tid];
                const double cs = csn[i * kHalf + tid], sn = csn[(j + i) * kHalf + tid];
                st.H[((size_t)i * m + j) * C + cc] = cs * a + sn * b;
                a = -sn * a + cs * b;
            }
            const double rr = hypot(a, hn);
            const double cs = rr > 0 ? a / rr : 1.0, sn = rr > 0 ? hn / rr : 0.0;
            st.H[((size_t)j * m + j) * C + cc] = rr;
            st.cs[(size_t)j * C + cc] = cs;
            st.sn[(size_t)j * C + cc] = sn;
            const double gj = st.g[(size_t)j * C + cc];
            st.g[(size_t)j * C + cc] = cs * gj;
            st.g[(size_t)(j + 1) * C + cc] = -sn * gj;
            st.kdim[cc] = j + 1;
            const double res = fabs(sn * gj);
            inv[tid] = hn > 0.0 ? 1.0 / hn : 0.0;
            if (res <= tol * st.bnorm[cc] || hn == 0.0 || j + 1 == m) st.active[cc] = 0;
        }
    }
    __syncthreads();
    const double sc = inv[c];
    double* Vn = V + (size_t)(j + 1) * g.vec;
    precondition(g, base, cell, z, [&](int row) { return sc != 0.0 ? w[base + (size_t)row * kLanes] * sc : 0.0; },
                 [&](int row, double v) { Vn[base + (size_t)row * kLanes] = v; });
}

// x += P (V y), y = H^-1 g over each cell's own Krylov dimension; iters += that dimension.
__global__ void __launch_bounds__(kVecThreads)
    k_update(Geo g, CellState st, const double* __restrict__ V, double* __restrict__ z, double* __restrict__ x,
             int* __restrict__ iters, int m) {
    __shared__ double y[kMaxBasis * kHalf];
    __shared__ int kmax;
    const int tid = threadIdx.x, c = tid % kHalf;
    const size_t cell = (size_t)blockIdx.x * kHalf + c;
    const size_t base = cell / kLanes * g.M * kLanes + cell % kLanes;
    if (tid == 0) kmax = 0;
    __syncthreads();
    const int kd = st.kdim[cell];
    if (tid < kHalf) {
        for (int i = kd - 1; i >= 0; --i) {
            double s = st.g[(size_t)i * g.C + cell];
            for (int l = i + 1; l < kd; ++l) s -= st.H[((size_t)i * m + l) * g.C + cell] * y[l * kHalf + c];
            const double d = st.H[((size_t)i * m + i) * g.C + cell];
            y[i * kHalf + c] = d != 0.0 ? s / d : 0.0;
        }
        if (cell < (size_t)g.n_cells) iters[cell] += kd;
        atomicMax(&kmax, kd);
    }
    __syncthreads();
    if (kmax == 0) return;
    precondition(
        g, base, cell, z,
        [&](int row) {
            double s = 0.0;
            const double* col = V + base + (size_t)row * kLanes;
            for (int i0 = 0; i0 < kd; i0 += 8) {
                double v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = col[(size_t)min(i0 + i, kd - 1) * g.vec];
#pragma unroll
                for (int i = 0; i < 8; ++i) s = fma(i0 + i < kd ? y[(i0 + i) * kHalf + c] : 0.0, v[i], s);
            }
            return s;
        },
        [](int, double) {});
    // the same thread wrote z's rows of its q
    for (int q = tid / kHalf; q < g.nq; q += kRowGroups)
        for (int a = 0; a < g.K; ++a) {
            const size_t at = base + (size_t)(q * g.K + a) * kLanes;
            x[at] += z[at];
        }
}

// The active cells in order: list[i], pos[cell] = i, and their number.
__global__ void __launch_bounds__(1024) k_list(const int* __restrict__ active, int n, int* __restrict__ list,
                                               int* __restrict__ pos, int* __restrict__ count) {
    __shared__ int warps[32];
    __shared__ int done;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) done = 0;
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int c = c0 + tid;
        const bool a = c < n && active[c];
        const unsigned ball = __ballot_sync(0xffffffffu, a);
        if (lane == 0) warps[warp] = __popc(ball);
        __syncthreads();
        int before = done;
        for (int w = 0; w < warp; ++w) before += warps[w];
        if (a) {
            const int i = before + __popc(ball & ((1u << lane) - 1));
            list[i] = c;
            pos[c] = i;
        }
        __syncthreads();
        if (tid == 0)
            for (int w = 0; w < 32; ++w) done += warps[w];
        __syncthreads();
    }
    if (tid == 0) *count = done;
}

// Gather the listed cells of two tiled vectors into whole tiles (zeros past the last cell); a block per tile in x, whose
// number has no limit of 65535.
__global__ void __launch_bounds__(256) k_gather(const double* __restrict__ a, const double* __restrict__ b,
                                                double* __restrict__ ga, double* __restrict__ gb,
                                                const int* __restrict__ list, int n, int M) {
    const int lane = threadIdx.x & 31, tile = blockIdx.x, i = tile * kLanes + lane;
    const size_t cell = i < n ? list[i] : 0, src = cell / kLanes * M * kLanes + cell % kLanes;
    for (int r = blockIdx.y * 8 + (threadIdx.x >> 5); r < M; r += gridDim.y * 8) {
        const size_t dst = ((size_t)tile * M + r) * kLanes + lane;
        ga[dst] = i < n ? a[src + (size_t)r * kLanes] : 0.0;
        gb[dst] = i < n ? b[src + (size_t)r * kLanes] : 0.0;
    }
}

#define KCHECK(expr)                                                                                      \
    do {                                                                                                  \
        cudaError_t e_ = (expr);                                                                          \
        if (e_ != cudaSuccess) {                                                                          \
            char m_[256];                                                                                 \
            snprintf(m_, sizeof(m_), "%s: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
            cf_set_last_error(m_);                                                                        \
            return e_ == cudaErrorMemoryAllocation ? CF_ENOMEM : CF_ECUDA;                                \
        }                                                                                                 \
    } while (0)

#define KLAUNCH() KCHECK(cudaGetLastError())

}  // namespace

extern "C" int cf_gmres_workspace_size(const cf_plan* plan, int64_t b, int32_t restart, size_t* bytes) {
    if (!plan || !bytes || b < 0 || restart < 1 || restart > 63) return CF_EINVAL;
    cf_plan_info info;
    int st = cf_plan_get_info(plan, &info);
    if (st != CF_OK) return st;
    const size_t nt = (size_t)((b + kLanes - 1) / kLanes);
    const size_t vec = nt * kLanes * (size_t)info.n_q * info.k;  // doubles per vector
    const size_t C = nt * kLanes;
    const size_t m = (size_t)restart;
    size_t d = vec * (m + 1)      // V
               + vec * 3          // w, z, J z
               + C * (m + 1) * m  // H
               + C * m * 2        // cs, sn
               + C * (m + 1)      // g
               + C * 2;           // bnorm, rel
    *bytes = d * sizeof(double) + C * 5 * sizeof(int) + 64 * sizeof(int) + 32 * 256;  // + alignment of 16 pieces
    return CF_OK;
}

extern "C" int cf_gmres_solve_tiled(cf_plan* plan, const double* f_t, double dt, const double* b_t, double* x_t,
                                    int64_t b, int32_t restart, int32_t max_iters, double tol,
                                    const double* precond, int32_t precond_per_cell, int32_t* iters_out,
                                    double* relres_out, void* workspace, size_t workspace_bytes, void* stream) {
    if (!plan || (b > 0 && (!f_t || !b_t || !x_t))) {
        cf_set_last_error("cf_gmres_solve_tiled: null argument");
        return CF_EINVAL;
    }
    if (restart < 1 || restart > 63 || max_iters < 1 || !(tol > 0)) {
        cf_set_last_error("cf_gmres_solve_tiled: restart must be in [1, 63], max_iters >= 1, tol > 0");
        return CF_EINVAL;
    }
    if (b == 0) return CF_OK;
    cf_plan_info info;
    int st = cf_plan_get_info(plan, &info);
    if (st != CF_OK) return st;
    size_t need = 0;
    st = cf_gmres_workspace_size(plan, b, restart, &need);
    if (st != CF_OK) return st;
    if (!workspace || workspace_bytes < need) {
        char msg[160];
        snprintf(msg, sizeof(msg), "cf_gmres_solve_tiled: workspace of %zu bytes, %zu needed", workspace_bytes, need);
        cf_set_last_error(msg);
        return CF_EINVAL;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int M = info.n_q * info.k;
    const int nt = (int)((b + kLanes - 1) / kLanes);
    const size_t C = (size_t)nt * kLanes;
    const size_t vec = C * M;
    const int m = restart;
    const int n_cells = (int)b;

    // carve the workspace
    char* p = (char*)workspace;
    auto take = [&](size_t nbytes) {
        char* q = p;
        p += (nbytes + 255) & ~size_t(255);
        return q;
    };
    double* V = (double*)take(vec * (m + 1) * sizeof(double));
    double* w = (double*)take(vec * sizeof(double));
    double* z = (double*)take(vec * sizeof(double));
    double* jz = (double*)take(vec * sizeof(double));
    CellState cs;
    cs.H = (double*)take(C * (m + 1) * m * sizeof(double));
    cs.cs = (double*)take(C * m * sizeof(double));
    cs.sn = (double*)take(C * m * sizeof(double));
    cs.g = (double*)take(C * (m + 1) * sizeof(double));
    cs.bnorm = (double*)take(C * sizeof(double));
    double* rel = (double*)take(C * sizeof(double));
    cs.kdim = (int*)take(C * sizeof(int));
    cs.active = (int*)take(C * sizeof(int));
    int* iters = (int*)take(C * sizeof(int));
    int* list = (int*)take(C * sizeof(int));
    int* pos = (int*)take(C * sizeof(int));
    int* counts = (int*)take(64 * sizeof(int));  // [0] cells above tol, [16] active cells
    if ((size_t)(p - (char*)workspace) > workspace_bytes) {
        cf_set_last_error("cf_gmres_solve_tiled: internal workspace layout overflow");
        return CF_EINVAL;
    }
    const Geo g{info.n_q, info.k, M, n_cells, C, vec, precond, precond_per_cell};
    const unsigned n_half = (unsigned)(C / kHalf);
    KCHECK(cudaMemsetAsync(iters, 0, C * sizeof(int), s));

    // out = J(f) u for n cells.  It runs on the q2 <-> q3 folded operator (the same bilinear form on half
    // the entries) when the operator folds, else on the plain one.
    int jv_mode = 2;
    auto apply_J = [&](double* out, const double* f, const double* u, int64_t n) -> int {
        KCHECK(cudaMemsetAsync(out, 0, (size_t)((n + kLanes - 1) / kLanes) * kLanes * M * sizeof(double), s));
        int rc = cf_jv_tiled(plan, out, f, u, n, jv_mode, s);
        if (rc == CF_EUNSUPPORTED && jv_mode == 2) {
            jv_mode = 0;
            cf_set_last_error("");
            rc = cf_jv_tiled(plan, out, f, u, n, jv_mode, s);
        }
        return rc;
    };

    k_bnorm<<<n_half, kVecThreads, 0, s>>>(g, b_t, cs.bnorm);
    KLAUNCH();

    int total = 0;
    int host_bad = n_cells;
    for (;;) {
        int rc = apply_J(jz, f_t, x_t, b);
        if (rc) return rc;
        KCHECK(cudaMemsetAsync(counts, 0, sizeof(int), s));
        k_residual<<<n_half, kVecThreads, 0, s>>>(g, cs, b_t, x_t, jz, w, V, z, dt, rel, counts, m, tol);
        KLAUNCH();
        KCHECK(cudaMemcpyAsync(&host_bad, counts, sizeof(int), cudaMemcpyDeviceToHost, s));
        KCHECK(cudaStreamSynchronize(s));
        if (host_bad == 0 || total >= max_iters) break;

        int n_active = n_cells;
        for (int j = 0; j < m && total < max_iters; ++j, ++total) {
            // J z of every cell, or, once a quarter of them are done, of the active ones alone, gathered into the
            // basis vectors that are still free (V_(j+2) on)
            const bool few = n_active < n_cells && 4 * (int64_t)n_active <= 3 * (int64_t)n_cells && j + 4 <= m;
            if (few) {
                double *fc = V + (size_t)(j + 2) * vec, *zc = fc + vec, *oc = zc + vec;
                const int nt_c = (n_active + kLanes - 1) / kLanes;
                k_gather<<<dim3((unsigned)nt_c, (unsigned)std::min(64, (M + 7) / 8)), 256, 0, s>>>(f_t, z, fc, zc, list,
                                                                                                  n_active, M);
                KLAUNCH();
                rc = apply_J(oc, fc, zc, n_active);
            } else {
                rc = apply_J(jz, f_t, z, b);
            }
            if (rc) return rc;
            auto step = j < 2    ? k_step<2>
                        : j < 4  ? k_step<4>
                        : j < 6  ? k_step<6>
                        : j < 8  ? k_step<8>
                        : j < 10 ? k_step<10>
                        : j < 12 ? k_step<12>
                                 : k_step<16>;
            step<<<n_half, kVecThreads, 0, s>>>(g, cs, V, w, z, few ? V + (size_t)(j + 4) * vec : jz, few ? pos : nullptr,
                                                dt, j, m, tol);
            KLAUNCH();
            k_list<<<1, 1024, 0, s>>>(cs.active, n_cells, list, pos, counts + 16);
            KLAUNCH();
            KCHECK(cudaMemcpyAsync(&n_active, counts + 16, sizeof(int), cudaMemcpyDeviceToHost, s));
            KCHECK(cudaStreamSynchronize(s));
            if (n_active <= 0) {
                ++total;
                break;
            }
        }
        k_update<<<n_half, kVecThreads, 0, s>>>(g, cs, V, z, x_t, iters, m);
        KLAUNCH();
    }
    if (iters_out) KCHECK(cudaMemcpyAsync(iters_out, iters, (size_t)n_cells * sizeof(int), cudaMemcpyDeviceToHost, s));
    if (relres_out) KCHECK(cudaMemcpyAsync(relres_out, rel, (size_t)n_cells * sizeof(double), cudaMemcpyDeviceToHost, s));
    KCHECK(cudaStreamSynchronize(s));
    if (host_bad > 0) {
        char msg[160];
        snprintf(msg, sizeof(msg), "cf_gmres_solve_tiled: %d of %d cells above tol after %d iterations", host_bad,
                 n_cells, total);
        cf_set_last_error(msg);
        return CF_ETIMEOUT;
    }
    return CF_OK;
}
