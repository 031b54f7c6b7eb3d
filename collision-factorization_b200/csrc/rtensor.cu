// rtensor.cu -- the reduced radial tensor R on the GPU.
//
// R_t[k1,k2,k3] is the reference's sum-factorised 5-D quadrature (compute_rtensor_sumfac_mex.cpp,
// 26 inputs prepared by GeneralCollisionTensor.m:43-181).  Its structure, restated:
//
//   for every radial node x and every "item" -- patch 1: (x, u) with an inner t loop; patch 2:
//   (x, y, t) -- the pre-collision speeds vL, vS and a Jacobian J fix the item; every inner point
//   (t, chi, eps) gives two post-collision velocities vp1, vp2, and for every channel t (an
//   l-triplet) the item accumulates
//     gain_s[k1] += W (sum_q Y_q(vp_s) P_gain[q]) * phi_{k1,l1}(|vp_s|)          (s = 1, 2)
//     loss_s[k1] += W' P_loss * phi_{k1,l1}(v_s)                                  (v_1 = vL, v_2 = vS)
//   and then contributes the rank-2 update
//     R_t[k1,k2,k3] += J (gain_1 - loss_1)[k1] phi_{k2,l2}(vL) phi_{k3,l3}(vS)
//                    + J (gain_2 - loss_2)[k1] phi_{k2,l2}(vS) phi_{k3,l3}(vL)
//   (phi_{k,l}(v) = norm_{k,l} L_k^{(l+1/2)}(v^2) v^l, Y the real spherical harmonics).
//
// On the device this is three kernels over chunks of items:
//   k_items     one CTA per job: an (x, u) item of patch 1 with all its t, or four items (x, y, t) of
//               patch 2.  A channel's valid q all lie in one band l1, so the sum over points is taken
//               once per (q, k) instead of once per channel:
//                   S_s[q][k] = sum_points W Y_q(vp_s) phi_{k,l(q)}(|vp_s|),
//               a [q x points] x [points x k] product per band on the FP64 tensor cores
//               (mma.sync m8n8k4), and gain_s[k1] = sum_q P_gain[q] S_s[q][k1] is taken once per
//               (item, t).  The threads evaluate harmonics and radial functions of up to 64 points per
//               side (vp_1, vp_2) at a time into shared memory, one thread per (velocity, function
//               family); azimuths come from x / rho and y / rho by rotation, without atan2 or sincos.
//               The CTA writes the items' "net" vectors J (gain - loss) and radial values at vL, vS;
//   k_contract  per channel and part of the chunk's items, R_t = sum net[k1] (phi (x) phi)[k2,k3] as a
//               [K x items] x [items x K^2] product on the same tensor cores;
//   k_reduce    adds the parts in a fixed order.
// Two exact simplifications are taken where the inputs allow them: (q, channel) pairs whose P_gain is
// zero everywhere are dropped (the reference's tables hold zeros for every sine harmonic), and then
// azimuths eps and -eps, whose cosine harmonics are equal, are merged into one node of both weights.
// Every R entry is summed in a fixed order, so the result is deterministic (the reference's
// OpenMP reduction order is not); it agrees with the reference to rounding.
// What bounds it: the barriers between its phases and the latency of its chains (square roots, quotients, exp and
// pow once per (item, t)): at L = 4, K = 5 issue slots 52 % full, FP64 pipe 15 % and its tensor part 9 %.
// Measured (B200, pad 20, device time): L = 4, K = 5 3.1 ms against 122 ms with per-channel sums at
// every point and a barrier pair per 16 points; L = 10, K = 8 124 ms against 1990 ms.  Patch-2 items in
// CTAs of 4 instead of one CTA per (x, y): 3.1 against 3.8 ms and 124 against 845 ms (a 48 MB chunk
// was less than one wave of CTAs).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "../../include/cf_b200.h"

void cf_set_last_error(const char* msg);

namespace {

constexpr int kItemThreads = 256;       // threads per k_items CTA
constexpr int kItemWarps = kItemThreads / 32;
constexpr int kMaxL = 31;               // N_Q = (L+1)^2 with L <= 31
constexpr int kMaxNK = 12;              // radial functions per l
constexpr double kEpsSafe = 1e-15;      // the reference's floor under square roots
constexpr double kPi = 3.14159265358979323846;

struct Dev {
    int NK, NL, NQ, L;
    double alpha;
    const double *x, *Wx;
    int Nx;
    const double *u1, *Wu1;
    int Nu1;
    const double *t1, *Wt1;
    int Nt1;
    const double *y2, *Wy2;
    int Ny2;
    const double *t2, *Wt2;
    int Nt2;
    const double *chi, *Wchi;
    int Nchi;
    const double *eps_c, *eps_s, *Weps;  // cos and sin of the eps nodes (host libm), weights
    int Neps;
    const double* rnorm;   // [NK x (L+1)]
    const double* shnorm;  // [NQ]
    const int *l1, *l2, *l3;
    const int* vq_begin;   // [NL+1] active (q, channel) pairs of each channel
    const int2* vq;        // per pair: row of S, column of the gain tables
    const int* slot;       // [NQ] harmonics slot of q, -1 where no pair uses q
    int n_slots, n_rows;   // used q; rows of S (distinct (q, l1))
    const int4* tiles;     // MMA tiles of S: (l, first row, rows <= 8, first k)
    const int* row_slot;   // [n_rows] harmonics slot of each row of S
    int n_tiles;
    int sine;              // some used q has m < 0
    const double* ploss1;  // [Nt1 x Nu1 x NL] as given
    const double* pgain1;  // [Nu1][Nt1][ld]
    const double* ploss2;  // [Ny2 x NL] as given
    const double* pgain2;  // [Ny2][ld]
    int64_t ld;
};

__device__ __forceinline__ void rt_dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// norm * L_k^{(l+1/2)}(v^2) * v^l for k = 0..NK-1 (three-term recurrence in k), out[k * stride]; vl = v^l
__device__ __forceinline__ void radial_l(int NK, int l, double v2, double vl, const double* rnorm,
                                         const double* inv, double* out, int stride) {
    const double al = (double)l + 0.5;
    double Lm = 1.0, Lc = 1.0 + al - v2;
    for (int k = 0; k < NK; ++k) {
        double Lk;
        if (k == 0) {
            Lk = 1.0;
        } else if (k == 1) {
            Lk = Lc;
        } else {
            Lk = ((2.0 * (k - 1) + 1.0 + al - v2) * Lc - ((k - 1) + al) * Lm) * inv[k];
            Lm = Lc;
            Lc = Lk;
        }
        out[(size_t)k * stride] = rnorm[k + NK * l] * Lk * vl;
    }
}

// What an (item, t) fixes; computed by one thread each, kPointBlock t at a time.
constexpr int kPointBlock = 32;
constexpr int kTBlock = 4;  // patch-2 items per CTA: a 48 MB chunk then is several waves of CTAs
struct Point {
    double cb_w;             // B Jt: the weight of every inner point
    double lw;               // the loss weight
    double vL, vS, Jo;
    double Ux[2], Uz[2], um[2], zx[2], zz[2];
};

__device__ void make_point(const Dev& d, int patch, int i, int o, int tt, Point& P) {
    const double xi = d.x[i];
    const double a = sqrt(xi / 2.0);
    double Jt, cb, umag, vL, vS, Jo;
    if (patch == 1) {
        const double u = d.u1[o], t = d.t1[tt];
        vL = a * (1.0 + u);
        vS = a * (1.0 - u);
        Jo = 0.5 * d.Wx[i] * d.Wu1[o] * u * exp(-xi * u * u) * (vL * vL * vS * vS);
        const double y = u * t;
        Jt = d.Wt1[tt] * (4.0 * u * t);
        cb = 1.0 - 2.0 * y * y;
        umag = sqrt(2.0 * xi) * u * sqrt(1.0 + (1.0 - u * u) * t * t);
    } else {
        const double y = d.y2[o], t = d.t2[tt];
        const double u = y * t;
        vL = a * (1.0 + u);
        vS = a * (1.0 - u);
        Jo = 0.5 * d.Wx[i] * d.Wy2[o] * y * (4.0 * y);
        Jt = d.Wt2[tt] * exp(-xi * u * u) * (vL * vL * vS * vS);
        cb = 1.0 - 2.0 * y * y;
        umag = sqrt(2.0 * xi) * y * sqrt(t * t + 1.0 - y * y * t * t);
    }
    const double sb = sqrt(fmax(1.0 - cb * cb, kEpsSafe));
    const double B = pow(umag * sqrt(2.0), d.alpha) / pow(xi, d.alpha / 2.0);
    P.lw = B * 2.0 * kPi * 2.0 * Jt;
    P.cb_w = B * Jt;
    P.vL = vL;
    P.vS = vS;
    P.Jo = Jo;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double vo = s == 0 ? vS : vL, vz = s == 0 ? vL : vS;
        P.Ux[s] = vo * sb;
        P.Uz[s] = vz + vo * cb;
        const double ux = -vo * sb, uz = vz - vo * cb;
        P.um[s] = sqrt(fmax(ux * ux + uz * uz, kEpsSafe));
        P.zx[s] = ux / P.um[s];
        P.zz[s] = uz / P.um[s];
    }
}

// The post-collision velocity of side s at inner point (chi n, eps e); returns |v| (floored).
__device__ __forceinline__ double post_velocity(const Dev& d, const Point& P, int s, int n, int e, double& vx,
                                                double& vy, double& vz) {
    const double cc = d.chi[n];
    const double sc = sqrt(fmax(1.0 - cc * cc, 0.0));
    const double upx = sc * d.eps_c[e], upy = sc * d.eps_s[e], upz = cc;
    const double rx = upx * P.zz[s] + upz * P.zx[s], rz = -upx * P.zx[s] + upz * P.zz[s];
    vx = 0.5 * (P.Ux[s] + P.um[s] * rx);
    vy = 0.5 * (P.um[s] * upy);
    vz = 0.5 * (P.Uz[s] + P.um[s] * rz);
    return sqrt(fmax(vx * vx + vy * vy + vz * vz, kEpsSafe));
}

// Shared layout of k_items for VS points per side and round (columns padded by 4 doubles: the MMA
// operands of a warp, 8 rows x 4 columns, then fall into distinct banks).
struct ItemLayout {
    int vs, ld;             // points per side and round; column stride
    int s_out;              // S in device memory: doubles per CTA (0: in shared memory)
    int parts;              // threads per (velocity, function family): they share out m or l
    size_t y, rv, s, rl, pts, tab, total;  // offsets in doubles
};

// Gain and loss accumulation of one job's items; writes the items' net vectors and radial values.
template <bool S_OUT>
__global__ void __launch_bounds__(kItemThreads)
    k_items(Dev d, ItemLayout lay, int64_t group0, int64_t n_groups, int64_t item0, int64_t n_items_chunk,
            double* __restrict__ net, double* __restrict__ radv, double* __restrict__ s_scratch) {
    extern __shared__ __align__(16) double sm[];
    const int NK = d.NK, L = d.L, NR = (L + 1) * NK;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int VS = lay.vs, LD = lay.ld;
    double* Y = sm + lay.y;      // [2][n_slots][LD]: W Y_q of the round's velocities
    double* RV = sm + lay.rv;    // [2][NR][LD]: radial functions of the round's velocities
    double* S = S_OUT ? s_scratch + (size_t)blockIdx.x * lay.s_out : sm + lay.s;  // [2][n_rows][NK]
    double* RL = sm + lay.rl;    // [2][NR]: radial functions at vL and vS
    Point* pts = reinterpret_cast<Point*>(sm + lay.pts);
    double* inv = sm + lay.tab;  // [32] 1 / n
    double* shn = inv + 32;      // [NQ]
    double* rno = shn + d.NQ;    // [NR]
    int* slot = reinterpret_cast<int*>(rno + NR);  // [NQ]

    // the launch's groups: patch-1 items first (a CTA each), then the (x, y) of patch 2, whose items go
    // kTBlock t to a CTA
    const int64_t n1 = (int64_t)d.Nx * d.Nu1;
    const int64_t here1 = max((int64_t)0, min(n1 - group0, n_groups));
    int patch, i, o, t_lo, t_hi;
    int64_t it0;  // patch 1: the item; patch 2: the item of t = 0
    if (blockIdx.x < here1) {
        const int64_t g = group0 + blockIdx.x;
        patch = 1;
        i = (int)(g / d.Nu1);
        o = (int)(g % d.Nu1);
        t_lo = 0;
        t_hi = d.Nt1;
        it0 = g;
    } else {
        const int n_tb = (d.Nt2 + kTBlock - 1) / kTBlock;
        const int64_t r = blockIdx.x - here1, j = group0 + here1 + r / n_tb - n1;
        patch = 2;
        i = (int)(j / d.Ny2);
        o = (int)(j % d.Ny2);
        t_lo = (int)(r % n_tb) * kTBlock;
        t_hi = min(d.Nt2, t_lo + kTBlock);
        it0 = n1 + j * d.Nt2;
    }
    for (int e = tid; e < 32; e += kItemThreads) inv[e] = e ? 1.0 / (double)e : 0.0;
    for (int e = tid; e < d.NQ; e += kItemThreads) {
        shn[e] = d.shnorm[e];
        slot[e] = d.slot[e];
    }
    for (int e = tid; e < NR; e += kItemThreads) rno[e] = d.rnorm[e];
    const int n_pts = d.Nchi * d.Neps;
    const int n_kg = (NK + 3) / 4, n_out = 2 * d.NL * n_kg;
    for (int tt = t_lo; tt < t_hi; ++tt) {
        if ((tt - t_lo) % kPointBlock == 0) {
            __syncthreads();
            for (int e = tid; e < min(kPointBlock, t_hi - tt); e += kItemThreads)
                make_point(d, patch, i, o, tt + e, pts[e]);
            __syncthreads();
        }
        const Point& P = pts[(tt - t_lo) % kPointBlock];
        const int64_t itl = it0 + (patch == 2 ? tt : 0) - item0;
        const bool first = patch == 2 || tt == 0;  // the item's first t
        for (int p0 = 0; p0 == 0 || p0 < n_pts; p0 += VS) {
            const int np = min(VS, n_pts - p0), np4 = (np + 3) & ~3;
            // harmonics of 2 np4 velocities, radial functions of the same, then (once per item)
            // the radial functions at vL and vS
            const int n_vel = lay.parts * 4 * np4;
            const int n_work = n_vel + (first && p0 == 0 ? 2 * (L + 1) : 0);
            for (int wi = tid; wi < n_work; wi += kItemThreads) {
                if (wi >= n_vel) {
                    const int e = wi - n_vel, s = e > L, l = e - s * (L + 1);
                    const double v = s ? P.vS : P.vL;
                    double vl = 1.0;
                    for (int j = 0; j < l; ++j) vl *= v;
                    radial_l(NK, l, v * v, vl, rno, inv, RL + s * NR + l * NK, 1);
                    continue;
                }
                const int role = wi >= n_vel / 2, w = wi - role * (n_vel / 2);
                const int part = w / (2 * np4), r = w - part * 2 * np4, s = r >= np4, c = r - s * np4;
                const int p = p0 + c;
                double vx = 0.0, vy = 0.0, vz = 0.0, vm = 0.0, W = 0.0;
                if (c < np) {
                    const int n = p / d.Neps, e = p % d.Neps;
                    vm = post_velocity(d, P, s, n, e, vx, vy, vz);
                    W = d.Wchi[n] * d.Weps[e];
                }
                if (role) {
                    double* out = RV + (size_t)s * NR * LD + c;
                    double vl = c < np ? 1.0 : 0.0;  // columns past the last point are zero
                    for (int l = 0; l <= L; ++l) {
                        if (l % lay.parts == part)
                            radial_l(NK, l, vm * vm, vl, rno, inv, out + (size_t)l * NK * LD, LD);
                        vl *= vm;
                    }
                } else {
                    double* out = Y + (size_t)s * d.n_slots * LD + c;
                    const double xc = c < np ? fmax(fmin(vz / vm, 1.0), -1.0) : 0.0;
                    const double st = sqrt(fmax((1.0 - xc) * (1.0 + xc), 0.0));
                    const double rho = sqrt(vx * vx + vy * vy);
                    const double cp = rho > 0.0 ? vx / rho : 1.0, sp = rho > 0.0 ? vy / rho : 0.0;
                    double pmm = W, cm = 1.0, sn = 0.0;  // the weight rides on P_mm
                    for (int m = 0; m <= L; ++m) {
                        if (m > 0) {
                            pmm *= -(2.0 * m - 1.0) * st;
                            const double c2 = cm * cp - sn * sp;
                            sn = sn * cp + cm * sp;
                            cm = c2;
                        }
                        if (m % lay.parts != part) continue;
                        double p_prev = 0.0, p_cur = pmm;
                        for (int l = m; l <= L; ++l) {
                            if (l == m + 1) {
                                p_prev = p_cur;
                                p_cur = xc * (2 * m + 1) * p_cur;
                            } else if (l > m) {
                                const double pn = (xc * (2 * l - 1) * p_cur - (l + m - 1) * p_prev) * inv[l - m];
                                p_prev = p_cur;
                                p_cur = pn;
                            }
                            const int q0 = l * l + l;
                            const int sc = slot[q0 + m];
                            if (sc >= 0) out[(size_t)sc * LD] = shn[q0 + m] * p_cur * cm;
                            if (d.sine && m > 0) {
                                const int ss = slot[q0 - m];
                                if (ss >= 0) out[(size_t)ss * LD] = shn[q0 - m] * p_cur * sn;
                            }
                        }
                    }
                }
            }
            __syncthreads();
            for (int j = warp; j < 2 * d.n_tiles; j += kItemWarps) {
                const int s = j >= d.n_tiles;
                const int4 t = d.tiles[j - s * d.n_tiles];  // l, first row, rows, first k
                const int ra = min(lane >> 2, t.z - 1), kb = min(t.w + (lane >> 2), NK - 1);
                const double* pa = Y + ((size_t)s * d.n_slots + d.row_slot[t.y + ra]) * LD + (lane & 3);
                const double* pb = RV + ((size_t)s * NR + t.x * NK + kb) * LD + (lane & 3);
                const int kc = t.w + 2 * (lane & 3);
                double* out = S + ((size_t)s * d.n_rows + t.y + (lane >> 2)) * NK + kc;
                const bool r_in = (lane >> 2) < t.z;
                const bool in0 = r_in && kc < NK, in1 = r_in && kc + 1 < NK;
                double c0 = 0.0, c1 = 0.0, e0 = 0.0, e1 = 0.0;
                if (p0 > 0) {
                    if (in0) c0 = out[0];
                    if (in1) c1 = out[1];
                }
                int g = 0;
                for (; g + 8 <= np4; g += 8) {
                    rt_dmma(c0, c1, pa[g], pb[g]);
                    rt_dmma(e0, e1, pa[g + 4], pb[g + 4]);
                }
                if (g < np4) rt_dmma(c0, c1, pa[g], pb[g]);
                if (in0) out[0] = c0 + e0;
                if (in1) out[1] = c1 + e1;
            }
            __syncthreads();
        }
        // net[s][k] of every channel: J (B Jt sum_q P_gain S - loss); a thread takes four k of one
        // (channel, side), so a pair's table entry and row number are read once for them, and owns
        // its outputs, so a patch-1 item's t add up in place
        const double* pgs = patch == 1 ? d.pgain1 + ((size_t)o * d.Nt1 + tt) * d.ld : d.pgain2 + (size_t)o * d.ld;
        for (int e = tid; e < n_out; e += kItemThreads) {
            const int ch = e / (2 * n_kg), r = e - ch * 2 * n_kg, s = r >= n_kg, k0 = (r - s * n_kg) * 4;
            const double* Ss = S + (size_t)s * d.n_rows * NK + k0;
            const int jb = d.vq_begin[ch], je = d.vq_begin[ch + 1];
            const double pl = patch == 1 ? d.ploss1[tt + (size_t)d.Nt1 * (o + (size_t)d.Nu1 * ch)]
                                         : d.ploss2[o + (size_t)d.Ny2 * ch];
            const double* rl = RL + s * NR + d.l1[ch] * NK + k0;
            const int nk = min(4, NK - k0);
            double g[4] = {0.0, 0.0, 0.0, 0.0};
            for (int j = jb; j < je; ++j) {
                const int2 rc = d.vq[j];
                const double w = pgs[rc.y];
                const double* row = Ss + (size_t)rc.x * NK;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < nk) g[k] += w * row[k];
            }
            double* dst = net + ((size_t)ch * n_items_chunk + itl) * 2 * NK + s * NK + k0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < nk) {
                    const double v = P.Jo * (P.cb_w * g[k] - P.lw * pl * rl[k]);
                    dst[k] = first ? v : dst[k] + v;
                }
        }
        if (first)
            for (int e = tid; e < 2 * NR; e += kItemThreads) radv[(size_t)itl * 2 * NR + e] = RL[e];
        __syncthreads();
    }
}

// part[split][channel][K^3] += the rank-2 updates of this split's items: an MMA per 4 items and term, A =
// net [k1 x items], B[item][k2 + K k3] = phi_{k2,l2} phi_{k3,l3} formed in the operand's lane.
constexpr int kContractThreads = 256;
constexpr int kContractWarps = kContractThreads / 32;
constexpr int kContractBlock = 64;                 // items staged per round
constexpr int kContractLd = kContractBlock + 4;    // conflict-free operand rows
template <int NK>
__global__ void __launch_bounds__(kContractThreads) k_contract(Dev d, const double* __restrict__ net,
                                                               const double* __restrict__ radv,
                                                               int64_t n_items_chunk, double* __restrict__ part) {
    constexpr int MT = (NK + 7) / 8, NT = (NK * NK + 7) / 8, K3 = NK * NK * NK;
    constexpr int kStage = 6 * NK * kContractLd;
    __shared__ double sm[kStage > K3 ? kStage : K3];
    double* sn = sm;                        // [2][NK][ld]: net vectors of the two sides
    double* sr = sm + 2 * NK * kContractLd; // [4][NK][ld]: vL at l2, vS at l3, vS at l2, vL at l3
    const int NR = (d.L + 1) * NK;
    const int ch = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int l2 = d.l2[ch], l3 = d.l3[ch];
    const int64_t i_lo = n_items_chunk * blockIdx.y / gridDim.y, i_hi = n_items_chunk * (blockIdx.y + 1) / gridDim.y;
    double c[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) c[m][n][0] = c[m][n][1] = 0.0;
    for (int64_t b0 = i_lo; b0 < i_hi; b0 += kContractBlock) {
        const int nb = (int)(i_hi - b0 < kContractBlock ? i_hi - b0 : kContractBlock);
        __syncthreads();
        for (int e = tid; e < kContractBlock * 2 * NK; e += kContractThreads) {
            const int it = e / (2 * NK), r = e % (2 * NK);
            sn[r * kContractLd + it] = it < nb ? net[((size_t)ch * n_items_chunk + b0 + it) * 2 * NK + r] : 0.0;
        }
        for (int e = tid; e < kContractBlock * 4 * NK; e += kContractThreads) {
            const int it = e / (4 * NK), r = e % (4 * NK), w = r / NK, k = r % NK;
            // w = 0: phi(vL) at l2; 1: phi(vS) at l3; 2: phi(vS) at l2; 3: phi(vL) at l3
            const int l = (w == 0 || w == 2) ? l2 : l3;
            const int side = (w == 0 || w == 3) ? 0 : 1;
            sr[r * kContractLd + it] = it < nb ? radv[(size_t)(b0 + it) * 2 * NR + side * NR + l * NK + k] : 0.0;
        }
        __syncthreads();
        for (int g = warp; g < 2 * (kContractBlock / 4); g += kContractWarps) {
            const int side = g & 1, it = (g >> 1) * 4 + (lane & 3);
            if ((g >> 1) * 4 >= nb) continue;
            double a[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int k1 = 8 * m + (lane >> 2);
                a[m] = k1 < NK ? sn[(side * NK + k1) * kContractLd + it] : 0.0;
            }
            const double* p2 = sr + (size_t)(2 * side) * NK * kContractLd + it;
            const double* p3 = p2 + NK * kContractLd;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int kk = 8 * n + (lane >> 2);
                const int k2 = kk % NK, k3 = min(kk / NK, NK - 1);
                const double b = p2[k2 * kContractLd] * p3[k3 * kContractLd];
#pragma unroll
                for (int m = 0; m < MT; ++m) rt_dmma(c[m][n][0], c[m][n][1], a[m], b);
            }
        }
    }
    // the warps' sums, added in warp order
    for (int w = 0; w < kContractWarps; ++w) {
        __syncthreads();
        if (warp == w) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int k1 = 8 * m + (lane >> 2), kk = 8 * n + 2 * (lane & 3) + h;
                        if (k1 < NK && kk < NK * NK) {
                            double* p = sm + k1 + NK * kk;
                            *p = w == 0 ? c[m][n][h] : *p + c[m][n][h];
                        }
                    }
        }
    }
    __syncthreads();
    double* dst = part + ((size_t)blockIdx.y * d.NL + ch) * K3;
    for (int e = tid; e < K3; e += kContractThreads) dst[e] += sm[e];
}

// R = the splits' sums in order.
__global__ void __launch_bounds__(256) k_reduce(const double* __restrict__ part, int n_split, int64_t n,
                                                double* __restrict__ R) {
    const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (e >= n) return;
    double s = part[e];
    for (int j = 1; j < n_split; ++j) s += part[(size_t)j * n + e];
    R[e] = s;
}

// dst[c * rows + r] = src[r * cols + c]: the gain tables from pair-major rows to slice-major rows.
__global__ void __launch_bounds__(256) k_transpose(const double* __restrict__ src, int64_t rows, int64_t cols,
                                                   double* __restrict__ dst) {
    __shared__ double t[32][33];
    const int64_t c0 = (int64_t)blockIdx.x * 32;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    for (int64_t r0 = (int64_t)blockIdx.y * 32; r0 < rows; r0 += (int64_t)gridDim.y * 32) {
        for (int j = y; j < 32; j += 8)
            if (r0 + j < rows && c0 + x < cols) t[j][x] = src[(r0 + j) * cols + c0 + x];
        __syncthreads();
        for (int j = y; j < 32; j += 8)
            if (c0 + j < cols && r0 + x < rows) dst[(c0 + j) * rows + r0 + x] = t[x][j];
        __syncthreads();
    }
}

typedef void (*ContractFn)(Dev, const double*, const double*, int64_t, double*);
ContractFn contract_for(int nk) {
    static const ContractFn fn[kMaxNK] = {k_contract<1>, k_contract<2>, k_contract<3>,  k_contract<4>,
                                          k_contract<5>, k_contract<6>, k_contract<7>,  k_contract<8>,
                                          k_contract<9>, k_contract<10>, k_contract<11>, k_contract<12>};
    return fn[nk - 1];
}

#define RT_CHECK(expr)                                                                                  \
    do {                                                                                                \
        cudaError_t e_ = (expr);                                                                        \
        if (e_ != cudaSuccess) {                                                                        \
            char m_[256];                                                                               \
            snprintf(m_, sizeof(m_), "%s: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
            cf_set_last_error(m_);                                                                      \
            st = e_ == cudaErrorMemoryAllocation ? CF_ENOMEM : CF_ECUDA;                                \
            goto done;                                                                                  \
        }                                                                                               \
    } while (0)

// The channels (l-triplets) and the CSR of their valid q_i (the reference stops each list at its
// first -1), after checking the sizes and indices of the inputs.
struct Channels {
    std::vector<int> l1, l2, l3, vq_begin, vq_q;
};

int sumfac_channels(const char* fn, double* R_out, const cf_sumfac_inputs* in, int32_t device, Channels& chn) {
    char msg[160];
    if (!R_out || !in) {
        snprintf(msg, sizeof(msg), "%s: null argument", fn);
        cf_set_last_error(msg);
        return CF_EINVAL;
    }
    const int NK = in->k_max + 1, NL = in->n_l, NQ = in->n_q;
    const int L = (int)std::lround(std::sqrt((double)NQ)) - 1;
    if (in->k_max < 0 || NK > 12 || NL < 1 || NQ < 1 || (L + 1) * (L + 1) != NQ || L > kMaxL || in->n_x < 1 ||
        in->n_u1 < 0 || in->n_t1 < 0 || in->n_y2 < 0 || in->n_t2 < 0 || in->n_chi < 0 || in->n_eps < 0) {
        snprintf(msg, sizeof(msg), "%s: sizes out of range (K_max+1 <= 12, N_Q = (L+1)^2 with L <= 31)", fn);
        cf_set_last_error(msg);
        return CF_ESHAPE;
    }
    const double* arrays[] = {in->x_nodes, in->w_x, in->radial_norm, in->sh_norm, in->l_triplets, in->qi_valid};
    for (const double* p : arrays)
        if (!p) {
            snprintf(msg, sizeof(msg), "%s: null input array", fn);
            cf_set_last_error(msg);
            return CF_EINVAL;
        }
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev == 0) {
        snprintf(msg, sizeof(msg), "%s: no CUDA device", fn);
        cf_set_last_error(msg);
        return CF_ENODEVICE;
    }
    if (device < 0 || device >= n_dev) return CF_EINVAL;

    std::vector<int>&l1 = chn.l1, &l2 = chn.l2, &l3 = chn.l3, &vq_begin = chn.vq_begin, &vq_q = chn.vq_q;
    l1.assign(NL, 0);
    l2.assign(NL, 0);
    l3.assign(NL, 0);
    vq_begin.assign(NL + 1, 0);
    vq_q.clear();
    for (int ch = 0; ch < NL; ++ch) {
        l1[ch] = (int)in->l_triplets[ch];
        l2[ch] = (int)in->l_triplets[ch + NL];
        l3[ch] = (int)in->l_triplets[ch + 2 * NL];
        if (l1[ch] < 0 || l1[ch] > L || l2[ch] < 0 || l2[ch] > L || l3[ch] < 0 || l3[ch] > L) {
            snprintf(msg, sizeof(msg), "%s: an l-triplet is outside 0..L", fn);
            cf_set_last_error(msg);
            return CF_EBADIDX;
        }
        for (int idx = 0; idx < NQ; ++idx) {
            const int q = (int)in->qi_valid[idx + (size_t)NQ * ch];
            if (q == -1) break;
            if (q < 1 || q > NQ) {
                snprintf(msg, sizeof(msg), "%s: qi_valid holds an index outside 1..N_Q", fn);
                cf_set_last_error(msg);
                return CF_EBADIDX;
            }
            vq_q.push_back(q - 1);
        }
        vq_begin[ch + 1] = (int)vq_q.size();
    }
    return CF_OK;
}

// The gain tables of a run: `slices` [n_slices][n_pairs] as given (the packed entry), or `pairs`
// [n_pairs][n_slices] rows picked from the dense tables, turned into slices on the device.
struct GainTable {
    const double* data = nullptr;
    int64_t n_slices = 0;
    bool pair_major = false;
};

// The quadrature proper.  pairs (used_col): for every active (q, channel) pair, in channel order, its
// column in the gain tables; vq_begin, vq_q: their CSR by channel.
int sumfac_run(double* R_out, const cf_sumfac_inputs* in, const Channels& chn, const std::vector<int>& vq_begin,
               const std::vector<int>& vq_q, const std::vector<int>& used_col, int64_t ld, const GainTable& g1,
               const GainTable& g2, int32_t device, double* device_seconds) {
    const int NK = in->k_max + 1, NL = in->n_l, NQ = in->n_q;
    const int L = (int)std::lround(std::sqrt((double)NQ)) - 1;
    const int n_pairs = (int)vq_q.size();

    // rows of S: the distinct (l1, q) of the active pairs, band by band; harmonics slots: the distinct q
    std::vector<std::vector<int>> band_q(L + 1);
    std::vector<int> slot(NQ, -1);
    int n_slots = 0, sine = 0;
    std::vector<std::vector<int>> band_row(L + 1, std::vector<int>(NQ, -1));
    for (int ch = 0; ch < NL; ++ch)
        for (int j = vq_begin[ch]; j < vq_begin[ch + 1]; ++j) {
            const int q = vq_q[j], l = chn.l1[ch];
            if (slot[q] < 0) slot[q] = n_slots++;
            if (band_row[l][q] < 0) {
                band_row[l][q] = 0;
                band_q[l].push_back(q);
            }
            int lq = (int)std::sqrt((double)q);
            while ((lq + 1) * (lq + 1) <= q) ++lq;
            while (lq * lq > q) --lq;
            if (q < lq * lq + lq) sine = 1;
        }
    std::vector<int4> tiles;
    std::vector<int> row_slot;
    for (int l = 0; l <= L; ++l) {
        std::sort(band_q[l].begin(), band_q[l].end());
        const int row0 = (int)row_slot.size(), n = (int)band_q[l].size();
        for (int r = 0; r < n; ++r) {
            band_row[l][band_q[l][r]] = row0 + r;
            row_slot.push_back(slot[band_q[l][r]]);
        }
        for (int r = 0; r < n; r += 8)
            for (int k = 0; k < NK; k += 8) tiles.push_back(make_int4(l, row0 + r, std::min(8, n - r), k));
    }
    const int n_rows = (int)row_slot.size();
    std::vector<int2> vq(n_pairs);
    for (int ch = 0; ch < NL; ++ch)
        for (int j = vq_begin[ch]; j < vq_begin[ch + 1]; ++j)
            vq[j] = make_int2(band_row[chn.l1[ch]][vq_q[j]], used_col[j]);

    // azimuth nodes; eps and -eps merged where only cosine harmonics are used (they see the same values)
    std::vector<double> eps_c, eps_s, w_eps;
    for (int e = 0; e < in->n_eps; ++e) {
        const double c = std::cos(in->eps[e]), sn = std::sin(in->eps[e]);
        bool merged = false;
        for (size_t j = 0; !sine && j < eps_c.size() && !merged; ++j)
            if (std::fabs(eps_c[j] - c) <= 1e-15 && std::fabs(eps_s[j] + sn) <= 1e-15) {
                w_eps[j] += in->w_eps[e];
                merged = true;
            }
        if (merged) continue;
        eps_c.push_back(c);
        eps_s.push_back(sn);
        w_eps.push_back(in->w_eps[e]);
    }

    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    int st = CF_OK;
    char* arena = nullptr;
    Dev d{};
    double *net = nullptr, *radv = nullptr, *dR = nullptr, *part = nullptr, *turn = nullptr;
    double *dg1 = nullptr, *dg2 = nullptr, *s_scratch = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    const int NR = (L + 1) * NK;
    // an item of patch 1 without t nodes adds nothing
    const int64_t n1 = in->n_t1 > 0 ? (int64_t)in->n_x * in->n_u1 : 0;
    const int64_t j2 = (int64_t)in->n_x * in->n_y2;
    const int64_t n_groups = n1 + (in->n_t2 > 0 ? j2 : 0);
    const size_t K3 = (size_t)NK * NK * NK, nR = K3 * NL;
    int max_smem = 0, n_sms = 0;
    ItemLayout lay{};
    size_t smem = 0;
    int64_t chunk = 0;
    int n_split = 1;
    std::vector<char> small;
    ContractFn contract = contract_for(NK);
    auto items = k_items<false>;
    d.NK = NK;
    d.NL = NL;
    d.NQ = NQ;
    d.L = L;
    d.alpha = in->alpha;
    d.Nx = in->n_x;
    d.Nu1 = n1 > 0 ? in->n_u1 : 0;
    d.Nt1 = in->n_t1;
    d.Ny2 = in->n_y2;
    d.Nt2 = in->n_t2;
    d.Nchi = in->n_chi;
    d.Neps = (int)eps_c.size();
    d.n_slots = n_slots;
    d.n_rows = n_rows;
    d.n_tiles = (int)tiles.size();
    d.sine = sine;
    d.ld = ld;
    RT_CHECK(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    RT_CHECK(cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, device));
    {
        // points per round: as many as the job has, up to 64; halved while that lets one more CTA stay
        // on the SM (phases of different CTAs overlap) and each round still fills the MMA steps
        const int n_pts = d.Nchi * d.Neps;
        auto layout = [&](int vs, int pad = 4, bool s_out = false) {
            ItemLayout y{};
            y.vs = vs;
            y.ld = vs + pad;
            y.s_out = s_out ? 2 * std::max(n_rows, 1) * NK : 0;
            y.parts = std::max(1, std::min(8, kItemThreads / (4 * vs)));
            size_t o = 0;
            y.y = o;
            o += (size_t)2 * std::max(n_slots, 1) * y.ld;
            y.rv = o;
            o += (size_t)2 * NR * y.ld;
            y.s = o;
            o += s_out ? 0 : (size_t)2 * std::max(n_rows, 1) * NK;
            y.rl = o;
            o += (size_t)2 * NR;
            y.pts = o;
            o += (size_t)kPointBlock * sizeof(Point) / sizeof(double);
            y.tab = o;
            o += 32 + (size_t)NQ + NR + (NQ + 1) / 2;
            y.total = o * sizeof(double);
            return y;
        };
        int vs = 64;
        while (vs > 4 && vs / 2 >= n_pts) vs /= 2;
        while (vs > 4 && layout(vs).total + 1024 > (size_t)max_smem) vs /= 2;
        while (vs > 16 && layout(vs).total > ((size_t)110 << 10)) vs /= 2;
        lay = layout(vs);
        // operators whose tables do not fit so: columns without padding (bank conflicts), then S in device memory (any
        // list of valid q, e.g. every q in every channel, or all harmonics at L = 23, K = 12)
        for (int way = 1; way <= 2 && lay.total + 1024 > (size_t)max_smem; ++way) lay = layout(4, 0, way == 2);
        smem = lay.total;
        if (lay.s_out) items = k_items<true>;
    }
    if (smem + 1024 > (size_t)max_smem) {
        cf_set_last_error("cf_rtensor_sumfac: N_Q too large for the shared-memory layout");
        st = CF_EUNSUPPORTED;
        goto done;
    }
    // chunk of items: the net vectors of a chunk (written by k_items, read once by k_contract) stay
    // within 48 MB, so they live in the 126 MB L2 between the two kernels instead of crossing HBM
    chunk = std::max<int64_t>(std::max<int64_t>(1, in->n_t2), ((int64_t)48 << 20) / ((int64_t)NL * 2 * NK * 8));
    chunk = std::min<int64_t>(chunk, n1 + j2 * std::max(in->n_t2, 0));
    if (lay.s_out) chunk = std::min<int64_t>(chunk, ((int64_t)256 << 20) / ((int64_t)lay.s_out * 8));  // a CTA per item at most
    chunk = std::max<int64_t>(chunk, std::max<int64_t>(1, in->n_t2));
    n_split = std::max(1, std::min(64, (4 * n_sms + NL - 1) / NL));
    {
        // one arena: the small inputs first (one copy), then the tables and the work buffers
        std::vector<std::pair<const void**, size_t>> where;
        auto add = [&](const void** dst, const void* src, size_t n_bytes) {
            const size_t at = small.size();
            small.resize((at + std::max<size_t>(n_bytes, 1) + 255) & ~(size_t)255);
            if (n_bytes) std::memcpy(small.data() + at, src, n_bytes);
            where.push_back({dst, at});
        };
        const size_t D = sizeof(double);
#define RT_ADD(dst, src, n) add((const void**)&(dst), (src), (n))
        RT_ADD(d.x, in->x_nodes, in->n_x * D);
        RT_ADD(d.Wx, in->w_x, in->n_x * D);
        RT_ADD(d.u1, in->u1_nodes, in->n_u1 * D);
        RT_ADD(d.Wu1, in->w_u1, in->n_u1 * D);
        RT_ADD(d.t1, in->t1_nodes, in->n_t1 * D);
        RT_ADD(d.Wt1, in->w_t1, in->n_t1 * D);
        RT_ADD(d.y2, in->y2_nodes, in->n_y2 * D);
        RT_ADD(d.Wy2, in->w_y2, in->n_y2 * D);
        RT_ADD(d.t2, in->t2_nodes, in->n_t2 * D);
        RT_ADD(d.Wt2, in->w_t2, in->n_t2 * D);
        RT_ADD(d.chi, in->mu_chi, in->n_chi * D);
        RT_ADD(d.Wchi, in->w_chi, in->n_chi * D);
        RT_ADD(d.eps_c, eps_c.data(), eps_c.size() * D);
        RT_ADD(d.eps_s, eps_s.data(), eps_s.size() * D);
        RT_ADD(d.Weps, w_eps.data(), w_eps.size() * D);
        RT_ADD(d.rnorm, in->radial_norm, (size_t)NR * D);
        RT_ADD(d.shnorm, in->sh_norm, (size_t)NQ * D);
        RT_ADD(d.l1, chn.l1.data(), NL * sizeof(int));
        RT_ADD(d.l2, chn.l2.data(), NL * sizeof(int));
        RT_ADD(d.l3, chn.l3.data(), NL * sizeof(int));
        RT_ADD(d.vq_begin, vq_begin.data(), vq_begin.size() * sizeof(int));
        RT_ADD(d.vq, vq.data(), vq.size() * sizeof(int2));
        RT_ADD(d.slot, slot.data(), slot.size() * sizeof(int));
        RT_ADD(d.tiles, tiles.data(), tiles.size() * sizeof(int4));
        RT_ADD(d.row_slot, row_slot.data(), row_slot.size() * sizeof(int));
#undef RT_ADD
        size_t total = small.size();
        auto room = [&](size_t n_doubles) {
            const size_t at = total;
            total = (total + std::max<size_t>(n_doubles, 1) * sizeof(double) + 255) & ~(size_t)255;
            return at;
        };
        const size_t nl1 = (size_t)in->n_t1 * in->n_u1 * NL, nl2 = (size_t)in->n_y2 * NL;
        const size_t ng1 = (size_t)g1.n_slices * ld, ng2 = (size_t)g2.n_slices * ld;
        const bool pm = g1.pair_major;
        const size_t o_l1 = room(nl1), o_l2 = room(nl2), o_g1 = room(ng1), o_g2 = room(ng2);
        const size_t o_net = room((size_t)chunk * NL * 2 * NK), o_rad = room((size_t)chunk * 2 * NR);
        const size_t o_R = room(nR), o_part = room((size_t)n_split * nR);
        // the pair-major rows are read before the work buffers are written
        const size_t o_s = room((size_t)chunk * lay.s_out);
        const size_t o_turn = pm ? room(std::max(ng1, ng2)) : 0;
        RT_CHECK(cudaMalloc((void**)&arena, total));
        for (auto& w : where) *w.first = arena + w.second;
        d.ploss1 = (double*)(arena + o_l1);
        d.ploss2 = (double*)(arena + o_l2);
        d.pgain1 = dg1 = (double*)(arena + o_g1);
        d.pgain2 = dg2 = (double*)(arena + o_g2);
        net = (double*)(arena + o_net);
        radv = (double*)(arena + o_rad);
        dR = (double*)(arena + o_R);
        part = (double*)(arena + o_part);
        s_scratch = (double*)(arena + o_s);
        turn = pm ? (double*)(arena + o_turn) : nullptr;
        RT_CHECK(cudaMemcpy(arena, small.data(), small.size(), cudaMemcpyHostToDevice));
        if (nl1) RT_CHECK(cudaMemcpy((double*)d.ploss1, in->p_loss_p1, nl1 * D, cudaMemcpyHostToDevice));
        if (nl2) RT_CHECK(cudaMemcpy((double*)d.ploss2, in->p_loss_p2, nl2 * D, cudaMemcpyHostToDevice));
        const GainTable* gs[2] = {&g1, &g2};
        double* dgs[2] = {dg1, dg2};
        for (int h = 0; h < 2; ++h) {
            const int64_t ns = gs[h]->n_slices;
            if (ns * ld == 0) continue;
            RT_CHECK(cudaMemcpy(pm ? turn : dgs[h], gs[h]->data, (size_t)ns * ld * D, cudaMemcpyHostToDevice));
            if (!pm) continue;
            const int64_t gx = (ns + 31) / 32, gy = std::min<int64_t>(65535, (ld + 31) / 32);
            k_transpose<<<dim3((unsigned)gx, (unsigned)gy), 256>>>(turn, ld, ns, dgs[h]);
            RT_CHECK(cudaGetLastError());
        }
    }
    RT_CHECK(cudaMemset(part, 0, (size_t)n_split * nR * sizeof(double)));
    RT_CHECK(cudaFuncSetAttribute(items, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    RT_CHECK(cudaEventCreate(&ev0));
    RT_CHECK(cudaEventCreate(&ev1));
    RT_CHECK(cudaEventRecord(ev0));
    for (int64_t g0 = 0; g0 < n_groups;) {
        // groups [g0, ge): patch-1 items, then as many whole (x, y) groups of patch 2 as the chunk still holds
        const int64_t nt2 = std::max(in->n_t2, 1);
        int64_t ge = g0 < n1 ? std::min(n1, g0 + chunk) : g0;
        const int64_t here1 = ge - g0;
        if (ge >= n1) ge = std::min(n_groups, ge + (chunk - here1) / nt2);
        const int64_t here2 = ge - g0 - here1;
        const int64_t i0 = g0 < n1 ? g0 : n1 + (g0 - n1) * nt2, nc = here1 + here2 * nt2;
        const int64_t ctas = here1 + here2 * ((nt2 + kTBlock - 1) / kTBlock);
        items<<<(unsigned)ctas, kItemThreads, smem>>>(d, lay, g0, ge - g0, i0, nc, net, radv, s_scratch);
        RT_CHECK(cudaGetLastError());
        contract<<<dim3((unsigned)NL, (unsigned)n_split), kContractThreads>>>(d, net, radv, nc, part);
        RT_CHECK(cudaGetLastError());
        g0 = ge;
    }
    k_reduce<<<(unsigned)((nR + 255) / 256), 256>>>(part, n_split, (int64_t)nR, dR);
    RT_CHECK(cudaGetLastError());
    RT_CHECK(cudaEventRecord(ev1));
    RT_CHECK(cudaEventSynchronize(ev1));
    if (device_seconds) {
        float ms = 0.f;
        RT_CHECK(cudaEventElapsedTime(&ms, ev0, ev1));
        *device_seconds = ms * 1e-3;
    }
    RT_CHECK(cudaMemcpy(R_out, dR, nR * sizeof(double), cudaMemcpyDeviceToHost));
done:
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    cudaFree(arena);
    cudaSetDevice(prev);
    return st;
}

// The (q, channel) pairs whose gain is zero everywhere add nothing and are dropped.
void keep_active(const Channels& chn, const std::vector<char>& active, std::vector<int>& begin, std::vector<int>& q,
                 std::vector<int>& col) {
    begin.assign(1, 0);
    q.clear();
    col.clear();
    for (size_t ch = 0; ch + 1 < chn.vq_begin.size(); ++ch) {
        for (int j = chn.vq_begin[ch]; j < chn.vq_begin[ch + 1]; ++j)
            if (active[j]) {
                q.push_back(chn.vq_q[j]);
                col.push_back(j);
            }
        begin.push_back((int)q.size());
    }
}

}  // namespace

extern "C" {

int cf_rtensor_sumfac(double* R_out, const cf_sumfac_inputs* in, int32_t device, double* device_seconds) {
    Channels chn;
    int st = sumfac_channels("cf_rtensor_sumfac", R_out, in, device, chn);
    if (st != CF_OK) return st;
    if (!in->p_gain_p1 || !in->p_gain_p2) {
        cf_set_last_error("cf_rtensor_sumfac: null input array");
        return CF_EINVAL;
    }
    // the active pairs' rows of the dense tables (contiguous in [t][u] and [y])
    const size_t NQ = in->n_q, n1 = (size_t)in->n_t1 * in->n_u1, n2 = in->n_y2;
    auto any = [](const double* p, size_t n) {
        for (size_t i = 0; i < n; ++i)
            if (!(p[i] == 0.0)) return true;
        return false;
    };
    const size_t nnz = chn.vq_q.size();
    std::vector<char> active(nnz, 0);
    auto row1 = [&](size_t ch, size_t j) { return in->p_gain_p1 + n1 * (chn.vq_q[j] + NQ * ch); };
    auto row2 = [&](size_t ch, size_t j) { return in->p_gain_p2 + n2 * (chn.vq_q[j] + NQ * ch); };
    for (size_t ch = 0; ch < (size_t)in->n_l; ++ch)
        for (int j = chn.vq_begin[ch]; j < chn.vq_begin[ch + 1]; ++j)
            active[j] = any(row1(ch, j), n1) || any(row2(ch, j), n2);
    std::vector<int> begin, q, col;
    keep_active(chn, active, begin, q, col);
    const size_t ld = q.size();
    std::vector<double> pg1(n1 * ld), pg2(n2 * ld);
    for (size_t ch = 0; ch < (size_t)in->n_l; ++ch)
        for (int a = begin[ch]; a < begin[ch + 1]; ++a) {
            std::copy(row1(ch, col[a]), row1(ch, col[a]) + n1, pg1.begin() + n1 * a);
            std::copy(row2(ch, col[a]), row2(ch, col[a]) + n2, pg2.begin() + n2 * a);
            col[a] = a;
        }
    GainTable g1, g2;
    g1.data = pg1.data();
    g1.n_slices = (int64_t)n1;
    g1.pair_major = true;
    g2.data = pg2.data();
    g2.n_slices = (int64_t)n2;
    g2.pair_major = true;
    return sumfac_run(R_out, in, chn, begin, q, col, (int64_t)ld, g1, g2, device, device_seconds);
}

int cf_rtensor_sumfac_packed(double* R_out, const cf_sumfac_inputs* in, const double* p_gain_p1_packed,
                             const double* p_gain_p2_packed, int32_t device, double* device_seconds) {
    Channels chn;
    int st = sumfac_channels("cf_rtensor_sumfac_packed", R_out, in, device, chn);
    if (st != CF_OK) return st;
    if (!p_gain_p1_packed || !p_gain_p2_packed) {
        cf_set_last_error("cf_rtensor_sumfac_packed: null packed gain table");
        return CF_EINVAL;
    }
    const size_t nnz = chn.vq_q.size(), n1 = (size_t)in->n_t1 * in->n_u1, n2 = in->n_y2;
    std::vector<char> active(nnz, 0);
    for (size_t i = 0; i < n1; ++i)
        for (size_t j = 0; j < nnz; ++j) active[j] |= !(p_gain_p1_packed[i * nnz + j] == 0.0);
    for (size_t i = 0; i < n2; ++i)
        for (size_t j = 0; j < nnz; ++j) active[j] |= !(p_gain_p2_packed[i * nnz + j] == 0.0);
    std::vector<int> begin, q, col;
    keep_active(chn, active, begin, q, col);
    GainTable g1, g2;
    g1.data = p_gain_p1_packed;
    g1.n_slices = (int64_t)n1;
    g2.data = p_gain_p2_packed;
    g2.n_slices = (int64_t)n2;
    return sumfac_run(R_out, in, chn, begin, q, col, (int64_t)nnz, g1, g2, device, device_seconds);
}

}  // extern "C"
