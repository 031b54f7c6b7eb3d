// outer_kernels.cuh -- angular-first kernels whose Phi step runs on the FP64 tensor cores.
//
// Per (t, q1) slice and cell, Phi = sum over the slice's runs of equal q2 of f(q2) (x) h, h = sum G f(q3),
// is a matrix product [K x runs] x [runs x K]: one mma.sync m8n8k4 takes four runs of one cell (K <= 8,
// padded to 8), with operands each lane reads straight from the cell's rows in shared memory.  A warp
// contracts one q1 row for four resident cells, and a team of warps one row for the unit's 16 (or 8):
//
//   * Phi step: for every chunk of four runs, lane (r = lane / 4, j = lane % 4) reads f(q2_j)[r] and forms
//     h_j[r] from one or two f(q3), two cells per 128-bit load; the cells are independent MMA chains.
//   * K^3 step: the MMA leaves each lane two Phi elements of every cell; lane partial sums acc[cell][k1]
//     += R[k1][k2][k3] Phi run over all slices of the row with the lane's 2 K values of R_t (x_R holds them in
//     lane order), and the lanes are summed once per row.
//   * R_t and the chunks of the next slices are copied (cp.async) into the team's ring by one of its warps in turn,
//     one named barrier per packet.
//
// Cells lie in shared memory in pairs, [pair][k][q][2], with the q rows padded to 4 modulo 8 pairs: the 8 lanes of
// a 128-bit phase (2 k x 4 runs) hit distinct banks when the runs' q are distinct modulo 4, which the host
// arranges when it packs runs into chunks (plan.cu, build_outer).  Empty slots of a chunk, and the second q3 of
// a run of one in a chunk of two, have G = 0 and read rows of zeros behind the last q: a product of zeros adds nothing,
// also where the slice's own f is infinite.
//
// What bounds it: shared-memory wavefronts (72 % of peak at L = 10, K = 8: 17 a cell and slice for the Phi operands,
// 8 for R_t, 8 for chunks, heads and copies), with the FP64 pipe at 50 %.  Four cells a warp (128 registers,
// 16 warps) rather than eight (255, 8 warps, half the R_t wavefronts): 1591 against 1847 us, latency; R_t read
// from L2 by each warp instead of staged: 2184 us.  B200, folded, L = 10, K = 8, 4096 cells: Q 1520 us (tile kernel
// 1624), J.v 2185 us (quarter-tile kernel 3060); L = 13, 1000 cells: Q 1057 us (1928); L = 10, 300 cells: 157 us (232).
#pragma once
#include <type_traits>

#include "launch.cuh"
#include "tile_kernels.cuh"

namespace cf {

// Work of one launch.  The units' rows, heaviest first, unit after unit, are one list that the CTAs share out in
// contiguous stretches of equal work (item_cum): at most two cut units a CTA, so teams run out of rows twice and f is
// staged little more than once.  Against whole units, then quarters, then sixteenths from a counter (B200, us):
// folded K = 8: L = 10, 4096 cells 1542 -> 1509, 300 cells 193 -> 158; L = 8, 2048 cells: J.v 543 -> 502; L = 13, 1000
// cells: 1120 -> 1045.  A streamed launch keeps quarters in order of arrival, so that every chunk gives work to all CTAs.
struct OuterSched {
    const int* bin_begin;  // as TileSched (streamed)
    const int* bin_q1;
    int n_units;           // of nc cells; streamed: each is taken in quarters
    int* counter;          // streamed
};

// Cell layout of one launch.
struct OuterGeom {
    int nc;     // cells per unit (16 or 8)
    int tiled;  // f, v, Q in the tiled layout; else the caller's cell-major arrays
};

__device__ __forceinline__ void outer_mma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

constexpr int kOuterChunk = 96;  // bytes of a chunk's slots: 4 x 16 (q2, q3a, q3b, -), 4 x (G_a, G_b)

struct OuterTask {
    int q1, s0, s1, pad;
    int4 first[2];  // x_slice[s0], x_slice[s0 + 1] (where the row has it)
};
template <int K, int G>
struct OuterStage {
    struct Slice {
        unsigned char R[K * 512];
        unsigned char chunks[kOuterChunks * kOuterChunk];
        int n2, n1, pad[2];  // chunks with two q3, chunks with one
    } sl[G];
    int4 next[G];  // x_slice entries after this packet's, as far as the row goes
    int task;      // < 0: no more packets
    int s;         // the slice after this packet's, or -1 where the row ends
    int a, b;      // slices (G > 1), or the one slice's n2 and n1
};

// Shared loads by 32-bit address.
__device__ __forceinline__ double2 lds2(uint32_t a) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}

__device__ __forceinline__ void team_sync(int team, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(team + 1), "r"(threads) : "memory");
}

// One warp of the team sends for the next packet: slices from s of the row `task`, entries `ent`, or, with
// s < 0, the first ones of the next row on the CTA's list.
template <int K, int G>
__device__ __forceinline__ void outer_feed(const DevOp& op, OuterStage<K, G>& st, int task, int s, const int4* ent,
                                           const OuterTask* tasks, int n_tasks, int* next, int lane) {
    if (s < 0) {
        if (lane == 0) task = atomicAdd(next, 1);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= n_tasks) {
            if (lane == 0) st.task = -1;
            return;
        }
        s = tasks[task].s0;
        ent = tasks[task].first;
    }
    const int s1 = tasks[task].s1, count = min(G, s1 - s);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (g >= count) break;
        const int4 sl = ent[g];
        const unsigned char* R = reinterpret_cast<const unsigned char*>(op.x_R) + (size_t)sl.x * K * 512 + lane * 16;
        unsigned char* dst = st.sl[g].R + lane * 16;
#pragma unroll
        for (int i = 0; i < K; ++i) cp_async16(dst + i * 512, R + i * 512);
        const unsigned char* ch = op.x_chunk + (size_t)sl.y * kOuterChunk;
        for (int i = lane; i < sl.w * (kOuterChunk / 16); i += 32) cp_async16(st.sl[g].chunks + i * 16, ch + i * 16);
        if (G > 1 && lane == 0) *reinterpret_cast<int2*>(&st.sl[g].n2) = make_int2(sl.z, sl.w - sl.z);
    }
    s += count;
    if (lane < G && s + lane < s1) cp_async16(st.next + lane, op.x_slice + s + lane);
    if (lane == 0)
        *reinterpret_cast<int4*>(&st.task) = G == 1 ? make_int4(task, s < s1 ? s : -1, ent[0].z, ent[0].w - ent[0].z)
                                                    : make_int4(task, s < s1 ? s : -1, count, 0);
    cp_async_commit();
}

// The rows a team takes from the CTA's list, for this warp's four cells (fw, vw: their rows).  out(task, sum) is
// called at a row's end with lane (c = lane / 8, k1 = lane % 8) holding Q[k1] of cell c.
template <int K, int NQP, bool JV, typename Out>
__device__ __forceinline__ void outer_rows(const DevOp& op, const double2* __restrict__ fw,
                                           const double2* __restrict__ vw, OuterStage<K, outer_group(NQP, JV)>* ring, int team,
                                           int team_warps, int w_in_team, const OuterTask* tasks, int n_tasks,
                                           int* next, int lane, Out out) {
    constexpr int C = kOuterCells, PS = outer_pair(K, NQP);
    const int j = lane & 3, r = lane >> 2;
    const uint32_t fr = (uint32_t)__cvta_generic_to_shared(fw) + min(r, K - 1) * NQP * 16;
    const uint32_t vr = JV ? (uint32_t)__cvta_generic_to_shared(vw) + min(r, K - 1) * NQP * 16 : 0;
    // Phi[k2 = r][k3 = 2 j, 2 j + 1]; rows and columns past K repeat others and are dropped
    const bool in0 = r < K && 2 * j < K, in1 = r < K && 2 * j + 1 < K;
    double acc[C][K];
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int k1 = 0; k1 < K; ++k1) acc[c][k1] = 0.0;

    constexpr int G = outer_group(NQP, JV);
    if (w_in_team == 0) outer_feed<K, G>(op, ring[0], 0, -1, nullptr, tasks, n_tasks, next, lane);
    int turn = 0;
    for (int b = 0;; b ^= 1) {
        // the packet is in (each warp waits for what it sent for), and every warp is done with the other one
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        team_sync(team, team_warps * 32);
        const OuterStage<K, G>& st = ring[b];
        const int4 hd = *reinterpret_cast<const int4*>(&st.task);
        const int task = hd.x;
        if (task < 0) break;
        if (w_in_team == turn) outer_feed<K, G>(op, ring[b ^ 1], task, hd.y, st.next, tasks, n_tasks, next, lane);
        turn = turn + 1 == team_warps ? 0 : turn + 1;
        const int count = G == 1 ? 1 : hd.z;
#pragma unroll 1
        for (int sg = 0; sg < count; ++sg) {
            const int2 nn = G == 1 ? make_int2(hd.z, hd.w) : *reinterpret_cast<const int2*>(&st.sl[sg].n2);
            double phi[C][2];
#pragma unroll
            for (int c = 0; c < C; ++c) phi[c][0] = phi[c][1] = 0.0;
            // a chunk of four runs, of one or two q3 each
            const unsigned char* ch = st.sl[sg].chunks;
            auto chunk = [&](auto two) {
                const uint2 qs = *reinterpret_cast<const uint2*>(ch + j * 8);  // byte offsets of q2, q3a, q3b in a row
                const double2 g = *reinterpret_cast<const double2*>(ch + 32 + j * 16);
                ch += kOuterChunk;
                const uint32_t o2 = qs.x & 0xffffu, oa = qs.x >> 16, ob = qs.y;
#pragma unroll
                for (int c = 0; c < C; c += 2) {
                    constexpr int P16 = PS * 16;
                    const double2 f2 = lds2(fr + o2 + c / 2 * P16), fa = lds2(fr + oa + c / 2 * P16);
                    double2 x = make_double2(g.x * fa.x, g.x * fa.y);
                    if constexpr (two) {
                        const double2 fb = lds2(fr + ob + c / 2 * P16);
                        x.x = fma(g.y, fb.x, x.x);
                        x.y = fma(g.y, fb.y, x.y);
                    }
                    if constexpr (JV) {
                        const double2 v2 = lds2(vr + o2 + c / 2 * P16), va = lds2(vr + oa + c / 2 * P16);
                        double2 y = make_double2(g.x * va.x, g.x * va.y);
                        if constexpr (two) {
                            const double2 vb = lds2(vr + ob + c / 2 * P16);
                            y.x = fma(g.y, vb.x, y.x);
                            y.y = fma(g.y, vb.y, y.y);
                        }
                        outer_mma(phi[c][0], phi[c][1], f2.x, y.x);
                        outer_mma(phi[c + 1][0], phi[c + 1][1], f2.y, y.y);
                        outer_mma(phi[c][0], phi[c][1], v2.x, x.x);
                        outer_mma(phi[c + 1][0], phi[c + 1][1], v2.y, x.y);
                    } else {
                        outer_mma(phi[c][0], phi[c][1], f2.x, x.x);
                        outer_mma(phi[c + 1][0], phi[c + 1][1], f2.y, x.y);
                    }
                }
            };
            for (int i = 0; i < nn.x; ++i) chunk(std::true_type{});
            for (int i = 0; i < nn.y; ++i) chunk(std::false_type{});
            if constexpr (K < 8) {
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    phi[c][0] = in0 ? phi[c][0] : 0.0;
                    phi[c][1] = in1 ? phi[c][1] : 0.0;
                }
            }
            const uint32_t Rl = (uint32_t)__cvta_generic_to_shared(st.sl[sg].R) + lane * 16;
#pragma unroll
            for (int k1 = 0; k1 < K; ++k1) {
                const double2 rr = lds2(Rl + k1 * 512);
#pragma unroll
                for (int c = 0; c < C; ++c) acc[c][k1] = fma(rr.y, phi[c][1], fma(rr.x, phi[c][0], acc[c][k1]));
            }
        }
        if (hd.y < 0) {
            // sum over the lanes by halving: lane bits 4, 3 pick the cell, bits 2, 1, 0 pick k1
            auto half = [&](double lo, double hi, int off) {
                const bool up = lane & off;
                return (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, off);
            };
            double x[8];
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) {
                if (k1 < K) {
                    const double y0 = half(acc[0][k1 < K ? k1 : 0], acc[2][k1 < K ? k1 : 0], 16);
                    const double y1 = half(acc[1][k1 < K ? k1 : 0], acc[3][k1 < K ? k1 : 0], 16);
                    x[k1] = half(y0, y1, 8);
                } else {
                    x[k1] = 0.0;
                }
            }
#pragma unroll
            for (int h = 4; h >= 1; h >>= 1)
#pragma unroll
                for (int i = 0; i < h; ++i) x[i] = half(x[i], x[i + h], h);
            out(task, x[0]);
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int k1 = 0; k1 < K; ++k1) acc[c][k1] = 0.0;
        }
    }
}

// Stage nc cells of one array into shared memory as [pair][k][q][cell of the pair].
template <int K, int NQP>
__device__ __forceinline__ void outer_stage(double* dst, const double* __restrict__ src, const OuterGeom& g, int n_q,
                                            long long cell0, long long n_cells, int warp, int lane) {
    constexpr int W = kOuterWarps, PS = outer_pair(K, NQP);
    if (g.tiled) {
        // rows of 32 cells; the unit's nc cells of 32 / nc rows per warp step
        const int sub = lane / g.nc, c = lane - sub * g.nc, step = 32 / g.nc;
        const double* tile = src + (size_t)(cell0 / CF_TILE) * n_q * K * CF_TILE + (cell0 % CF_TILE) + c;
        double* d = dst + (size_t)(c >> 1) * PS * 2 + (c & 1);
        for (int row = warp * step + sub; row < n_q * K; row += W * step)
            cp_async8(d + 2 * ((row % K) * NQP + row / K), tile + (size_t)row * CF_TILE);
    } else {
        const size_t M = (size_t)n_q * K;
        for (int row = warp; row < g.nc * K; row += W) {
            const int c = row / K, k = row % K;
            double* d = dst + 2 * ((size_t)(c >> 1) * PS + k * NQP) + (c & 1);
            if (cell0 + c < n_cells) {
                const double* s = src + (size_t)(cell0 + c) * M + (size_t)k * n_q;
                for (int q = lane; q < n_q; q += 32) cp_async8(d + 2 * q, s + q);
            } else {
                for (int q = lane; q < n_q; q += 32) d[2 * q] = 0.0;
            }
        }
    }
}

template <int K, int NQP, bool JV>
__global__ void __launch_bounds__(kOuterWarps * 32, 1)
    af_outer_kernel(DevOp op, OuterSched sc, OuterGeom g, StreamSync ss, const double* __restrict__ f,
                    const double* __restrict__ v, double* q, long long n_cells) {
    constexpr int W = kOuterWarps;
    extern __shared__ __align__(16) double smem[];
    __shared__ int s_unit, s_next;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double* fs = smem;
    double* vs = JV ? smem + (size_t)g.nc * outer_pair(K, NQP) : nullptr;
    // after the cells: the teams' rings, the tasks
    constexpr int G = outer_group(NQP, JV);
    OuterStage<K, G>* rings =
        reinterpret_cast<OuterStage<K, G>*>(smem + (size_t)(JV ? 2 : 1) * g.nc * outer_pair(K, NQP));
    static_assert(2 * sizeof(OuterStage<K, G>) == outer_ring_bytes(K, NQP, JV), "ring size");
    const int team_warps = g.nc / kOuterCells, team = warp / team_warps, w_in_team = warp - team * team_warps;
    OuterTask* tasks = reinterpret_cast<OuterTask*>(rings + 2 * (W / team_warps));
    const size_t mine = (size_t)w_in_team * (kOuterCells / 2) * outer_pair(K, NQP);  // this warp's cells
    // the rows of zeros, which staging leaves alone
    const int n_zero = outer_zeros(op.n_q, NQP);
    for (int i = tid; i < (JV ? 2 : 1) * (g.nc / 2) * K * n_zero; i += W * 32) {
        const int row = i / n_zero, pair = row / K;
        reinterpret_cast<double2*>(fs)[(size_t)pair * outer_pair(K, NQP) + row % K * NQP + op.n_q + i % n_zero] =
            make_double2(0.0, 0.0);
    }
    int staged = -1;
    // not streamed: what is left of this CTA's stretch, from row s_from.y of unit s_from.x to row s_to.y of unit s_to.x
    __shared__ int2 s_from, s_to;
    if (!ss.ready) {
        const int2 from = stretch_cut<W * 32>(op.item_cum, op.n_items, sc.n_units, blockIdx.x),
                   to = stretch_cut<W * 32>(op.item_cum, op.n_items, sc.n_units, blockIdx.x + 1);
        if (tid == 0) {
            s_from = from;
            s_to = to;
        }
        __syncthreads();
    }
    for (;;) {
        int ht, b0, nb;
        if (ss.ready) {
            if (tid == 0) s_unit = atomicAdd(sc.counter, 1);
            __syncthreads();
            if (s_unit >= 4 * sc.n_units) break;
            ht = s_unit / 4;
            const int bin = 1 + s_unit % 4;
            b0 = sc.bin_begin[bin];
            nb = sc.bin_begin[bin + 1] - b0;
        } else {
            ht = s_from.x;
            b0 = s_from.y;
            if (ht > s_to.x || (ht == s_to.x && b0 >= s_to.y)) break;
            nb = (ht == s_to.x ? s_to.y : op.n_items) - b0;
        }
        const int chunk = ss.ready ? ht / ss.ht_per_chunk : 0;
        const long long cell0 = (long long)ht * g.nc;
        if (ht != staged) {
            if (ss.ready) {
                if (tid == 0) {
                    const long long t0 = clock64();
                    while (ld_acquire(ss.ready + chunk) != ss.epoch) {
                        if (*reinterpret_cast<volatile int*>(ss.abort) == ss.epoch) break;
                        if (clock64() - t0 > ss.wait_cycles) {
                            *reinterpret_cast<volatile int*>(ss.abort) = ss.epoch;
                            *reinterpret_cast<volatile int*>(ss.err) = 1;
                            break;
                        }
                        __nanosleep(256);
                    }
                }
                __syncthreads();
            }
            outer_stage<K, NQP>(fs, f, g, op.n_q, cell0, n_cells, warp, lane);
            if constexpr (JV) outer_stage<K, NQP>(vs, v, g, op.n_q, cell0, n_cells, warp, lane);
            cp_async_commit();
            cp_async_wait_all();
            staged = ht;
        }
        if (tid == 0) s_next = 0;
        for (int i = tid; i < nb; i += W * 32) {
            OuterTask t;
            t.q1 = sc.bin_q1[b0 + i];
            t.s0 = op.x_q1[t.q1];
            t.s1 = op.x_q1[t.q1 + 1];
            t.pad = 0;
            t.first[0] = op.x_slice[t.s0];
            t.first[1] = op.x_slice[min(t.s0 + 1, t.s1 - 1)];
            tasks[i] = t;
        }
        __syncthreads();
        outer_rows<K, NQP, JV>(
            op, reinterpret_cast<const double2*>(fs) + mine, reinterpret_cast<const double2*>(vs) + (JV ? mine : 0),
            rings + 2 * team, team, team_warps, w_in_team, tasks, nb, &s_next, lane, [&](int task, double sum) {
                const int q1 = tasks[task].q1, k1 = lane & 7;
                const long long cell = cell0 + w_in_team * kOuterCells + (lane >> 3);
                if (k1 >= K || (!g.tiled && cell >= n_cells)) return;
                double* qp = g.tiled ? q + (((size_t)(cell / CF_TILE) * op.n_q + q1) * K + k1) * CF_TILE + cell % CF_TILE
                                     : q + (size_t)cell * op.n_q * K + (size_t)k1 * op.n_q + q1;
                *qp += sum;
            });
        if (ss.done) __threadfence();
        __syncthreads();
        if (!ss.ready) {
            if (tid == 0) s_from = make_int2(ht + 1, 0);
            __syncthreads();
        }
        if (tid == 0 && ss.done) {
            const int h0 = chunk * ss.ht_per_chunk;
            const int c_ht = min(ss.ht_per_chunk, sc.n_units - h0);
            const int c_units = c_ht * 4;  // a streamed launch cuts every half-tile into 4
            if (atomicAdd(ss.done + chunk, 1) == c_units - 1) {
                __threadfence_system();
                *reinterpret_cast<volatile int*>(ss.host_done + chunk) = ss.epoch;
            }
        }
    }
}

}  // namespace cf
