// launch.cuh -- per-K launch entry points.  Each K is instantiated in its own translation unit
// (inst_k<K>.cu) so the kernels compile in parallel; plan.cu calls them through cf_launch().
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace cf {

enum Op { OP_AF = 0, OP_RF = 1, OP_JV = 2 };

// Kernel families for the angular-first / Jacobian forms.
enum Path { PATH_AUTO = 0, PATH_GATHER = 1, PATH_TILE = 2, PATH_PAIR = 3, PATH_PAIR_L1 = 4, PATH_PAIR_SPLIT = 5, PATH_TILE_MMA = 6,
           PATH_BF16_MMA = 7 /* reported only: the BF16-split form's kernel */,
           PATH_TILE4 = 8 /* reported only: the quarter-tile kernel, where the 16-cell tile does not fit */,
           PATH_FEW = 9 /* reported only: the few-cell kernel (a handful of cells per call) */,
           PATH_SPLIT_I8 = 10 /* reported only: the exact-split form's kernel (split.cu) */,
           PATH_BAND = 11 /* the band kernels on the cell-major arrays (split.cu): the FP64 forms on request */,
           PATH_BAND_BF16 = 12 /* reported only: the BF16-split form on the band kernel (tcgen05, split.cu) */,
           PATH_RF_DENSE = 13 /* reported only: the radial-first dense form (rfdense.cu) */,
           PATH_LBLOCK = 14 /* the l-block kernel (split.cu): band units, f staged per l-triplet, K = 8 and 12 */,
           // the outer-product kernel on units of 16 and of 8 cells: cf_plan_info reports them as PATH_TILE and
           // PATH_TILE4, the families whose place it takes, cf_plan_last_kernel by their own name
           PATH_OUTER = 15, PATH_OUTER8 = 16 };

struct LaunchArgs {
    DevOp op;
    const double* fT;
    const double* vT;
    double* QT;
    int64_t n_tiles;
    int64_t n_cells;
    cudaStream_t stream;
    int what;    // Op
    bool exact;  // reference operation order, no FMA
    int path;    // Path
    // tile-resident kernels: q1 bins, work-queue counter, device limits
    const int* bin_begin;
    const int* bin_q1;
    int* counter;
    int n_sms;
    size_t max_smem;
    // pair kernels: bins over pair items, items (qa, qb)
    const int* pbin_item;
    const int2* pitems;
    const long long* pair_cum;  // [n_pitems + 1] work of the items pbin_item[0 .. i) added up
    int n_pitems;
    // FP32 form: tiled FP32 copies of f (and v) in place of fT / vT
    bool f32;
    const float* fT32;
    // automatic order for the fast Q form: false = pair kernel first, true = tile kernel first
    bool tile_first;
    // BF16-split form (f32 is set too: FP32 tiles of f)
    bool bf16;
    // streamed host path: the tile kernel on cell-major f and Q while they are copied in and out
    const StreamSync* ss = nullptr;
    const double* f_cm = nullptr;
    double* q_cm = nullptr;
    const double* v_cm = nullptr;  // the exact J.v above K = 8 (rows): v, cell-major like f_cm
    // a handful of cells: the few-cell kernel on cell-major f_cm and q_cm (status -1 where it does not apply);
    // with few_host_f / few_host_q set, f and Q_in are those host arrays, passed in the launch's
    // parameter block, and q_cm receives Q_out
    bool few = false;
    const double* few_host_f = nullptr;
    const double* few_host_q = nullptr;
    // FP32 J.v: tiled FP32 copy of v
    const float* vT32 = nullptr;
    // with few: the exact form of any number of cells on the row kernel (one CTA per (q1, pair of cells), on the
    // cell-major arrays), the exact route where the batch kernels' register tiles do not fit (K > 8)
    bool rows = false;
    // the fast FP64 forms on the pair kernel, on the cell-major arrays f_cm, v_cm, q_cm
    bool pair_cm = false;
};

// Status codes mirror cf_status: 0 ok, 5 CUDA error, 8 unsupported, 2 shape.
struct LaunchResult {
    int status;
    int launches;
    cudaError_t cuda;
    int path;  // the kernel family that ran
};

#define CF_DECLARE_K(KK) LaunchResult launch_k##KK(const LaunchArgs& a);
CF_DECLARE_K(1) CF_DECLARE_K(2) CF_DECLARE_K(3) CF_DECLARE_K(4) CF_DECLARE_K(5) CF_DECLARE_K(6)
CF_DECLARE_K(7) CF_DECLARE_K(8) CF_DECLARE_K(9) CF_DECLARE_K(10) CF_DECLARE_K(11) CF_DECLARE_K(12)
CF_DECLARE_K(13) CF_DECLARE_K(14) CF_DECLARE_K(15) CF_DECLARE_K(16)
#undef CF_DECLARE_K

// Lanes per cell (P) of the fast kernels: the K x K Phi accumulator is split over P lanes by
// k3 column once it no longer fits one lane's registers.
constexpr int af_P(int K) { return K <= 8 ? 1 : (K <= 12 ? 2 : 4); }
// Warps per CTA of the FP64 pair kernel: as many as the registers of a whole Phi per lane leave (Q at K = 5: 128 a
// lane; K = 6, and J.v at K = 5: 168; else 255, or several CTAs on an SM below K = 5).
constexpr int pair_W(int K, bool jv = false) { return K == 5 ? (jv ? 12 : 16) : (K == 6 && !jv ? 12 : 8); }
// Shared memory of a warp: R_t and, where registers are short (the 16- and 12-warp Q forms), the row sums.
constexpr bool pair_sums_shared(int W, bool jv) { return W > 8 && !jv; }
constexpr int pair_warp_doubles(int K, int W, bool jv) { return (K * K * K + 1) / 2 * 2 + (pair_sums_shared(W, jv) ? K * 32 : 0); }
// The FP64 pair kernel's warps where its 16-cell tile of f (and v) fits beside their copies of R_t: pair_W, or 8 where
// only these fit (Q at L = 17, K = 5 and at L = 15, K = 6); 0 where neither does.
constexpr int pair_fit(int n_q, int K, bool jv, size_t max_smem) {
    if (K > 8) return 0;
    for (int W : {pair_W(K, jv), 8})
        if (sizeof(double) * ((size_t)(jv ? 2 : 1) * n_q * K * 16 + (size_t)W * pair_warp_doubles(K, W, jv)) + 256 <= max_smem)
            return W;
    return 0;
}
// Whether the automatic order takes the pair kernel where it fits.  With 8 warps for want of room the gather kernel (folded,
// K = 5) and the tile kernel (plain, K = 6) are the faster ones on some batches (B200, us, pair / other): L = 17, K = 5 folded:
// 100 cells 422 / 529, 300: 923 / 853, 2048: 4859 / 4279 (plain 7850 / 8402); L = 15, K = 6 plain: 20 cells 400 / 292, 100:
// 493 / 431, 300: 1143 / 1137, 1000: 2984 / 3106.
constexpr bool pair_auto(int n_q, int K, bool folded, bool jv, int64_t n_cells, size_t max_smem) {
    if (jv || pair_fit(n_q, K, jv, max_smem) == pair_W(K, jv)) return true;
    return K % 2 ? !folded || n_cells <= 200 : n_cells > 300;
}
constexpr int kTileBufs = 4;  // half-tiles that a CTA of the tile kernel holds at a time, at most
// K that the outer-product kernels (outer_kernels.cuh) take.
constexpr bool outer_for(int K) { return K >= 7 && K <= 8; }

// Where they are taken: every fast form at these K but the plain J.v at K = 7 on batches of more than two thirds of a half-tile
// per SM, which stays on the pair kernel where that fits (it does not at L = 10: 2000 cells 1944 us, 3084 on the gather kernel
// otherwise).  But for that one form the kernel, and so a cell's bits, does not depend on the batch.
// The faster family (B200, us, outer / the better of tile and pair): on small batches at every size (20 cells, L = 3 17.4 /
// 17.4, L = 6 22.5 / 28.7, L = 10 39.9 / 57.5, K = 8 folded Q), on large ones from L = 8 on at K = 8 (4096 cells, folded Q: L = 8
// 705 / 711, L = 10 1520 / 1624; J.v L = 8 980 / 1009; plain Q L = 8 1254 / 1254, L = 10 2832 / 3011; L = 13, 1000 cells 1055 /
// 1928) and for the folded Q at K = 7 (646 / 668).  Below, the tile and pair kernels in stretches are the faster ones (4096
// cells, K = 8 folded Q: L = 6 290 / 261, L = 3 63 / 45; K = 7 plain Q: L = 5 253 / 191, L = 8 1150 / 982), but only
// from a hundred to six hundred cells on.
constexpr bool outer_takes(int n_q, int K, bool folded, bool jv, int64_t n_cells, int n_sms, size_t max_smem) {
    return outer_for(K) && (K == 8 || folded || !jv || (n_cells + 15) / 16 * 3 <= 2 * n_sms || pair_fit(n_q, K, true, max_smem) == 0);
}

// Shared-memory geometry of the outer-product kernels.  Cells lie in pairs, [pair][k][q][cell of the pair],
// with rows of NQP doubles per cell fixed at compile time (one of two widths, 4 modulo 8, so that the 8 lanes
// of a 128-bit load phase, 2 k x 4 q distinct modulo 4, hit distinct banks) and an odd pair stride.
constexpr int outer_nqp(int width) { return width == 0 ? 132 : 268; }  // L <= 10, L <= 15
// Rows of zeros behind the last q (at least one), which a chunk's empty places read: four where there is room, one
// for each residue modulo 4.
constexpr int kOuterZeros = 4;
constexpr int outer_zeros(int n_q, int nqp) { return nqp - n_q < kOuterZeros ? nqp - n_q : kOuterZeros; }
constexpr int outer_pair(int K, int nqp) { return K * nqp + 1; }       // 16-byte elements per pair of cells
constexpr int kOuterCells = 4;   // cells per warp: 128 registers a lane hold acc and Phi, 16 warps fit
constexpr int kOuterWarps = 16;
constexpr int kOuterChunks = 8;  // chunks of 4 runs per slice at most (longer slices are cut)
// A team's ring of two packets of up to outer_group() slices: R_t in lane order, the chunks, the heads.  Q takes
// two slices to a packet at the narrow width (half the team barriers: 1552 against 1591 us at L = 10, K = 8,
// 4096 cells); with f and v resident, or the wide rows, only one fits.
constexpr int outer_group(int nqp, bool jv) { return !jv && nqp == outer_nqp(0) ? 2 : 1; }
constexpr int outer_ring_bytes(int K, int nqp, bool jv) {
    return 2 * outer_group(nqp, jv) * (K * 512 + kOuterChunks * 96 + 32) + 32;
}
// nc cells of f (and v), a ring per team of nc / 4 warps, and a task per q1 row.
constexpr size_t outer_smem_bytes(int n_q, int K, int nqp, int nc, bool jv) {
    return (size_t)(jv ? 2 : 1) * (nc / 2) * outer_pair(K, nqp) * 16 +
           (size_t)(kOuterWarps * kOuterCells / nc) * outer_ring_bytes(K, nqp, jv) + (size_t)n_q * 48;
}
// The widest unit that fits: 16 cells per unit before 8; (width, cells), or cells = 0 where none does.
struct OuterFit {
    int width, nc;
};
constexpr OuterFit outer_fit(int n_q, int K, bool jv, size_t max_smem) {
    const int width = n_q < outer_nqp(0) ? 0 : 1;
    if (n_q >= outer_nqp(width)) return {0, 0};
    for (int nc = 16; nc >= 8; nc -= 8)
        if (outer_smem_bytes(n_q, K, outer_nqp(width), nc, jv) + 256 <= max_smem) return {width, nc};
    return {0, 0};
}
constexpr int jv_P(int K) { return K <= 6 ? 1 : (K <= 8 ? 2 : 4); }

}  // namespace cf
