// hf_cg.cuh -- device code that the persistent CG kernels share: wait limits, the tile's cells, a scene's scalars.
#pragma once

#include "hf_device.cuh"
#include "hf_kernels.cuh"

namespace hf {

constexpr unsigned long long kBarrierTimeoutNs = 2000000000ull;   // 2 s
// Limit of every bounded wait of the CG kernels (grid and lane barriers, TMA copies, tagged words), and the block that does
// not arrive at the first grid barrier (or first exchange) of each persistent CG launch (-1: none; kAbsentLate + b: block b
// of an on-chip pressure solve keeps its final pressures on shared faces to itself).  The defaults are what every solve
// uses; hf_set_wait_limit changes both, so that a test can make a wait run out on purpose and check that the kernel reports
// HF_SCENE_BARRIER_TIMEOUT and returns with the context usable.
static __constant__ unsigned long long c_wait_limit_ns = kBarrierTimeoutNs;
static __constant__ int c_absent_block = -1;
constexpr int kAbsentLate = 65536;

__device__ __forceinline__ int uidx_(int n, int i, int j, int k) { return (i * n + j) * n + k; }
__device__ __forceinline__ int vidx_(int n, int i, int j, int k) { return (i * (n + 1) + j) * n + k; }
__device__ __forceinline__ int widx_(int n, int i, int j, int k) { return (i * n + j) * (n + 1) + k; }

// cell m (0..3) of thread lt in a tile
struct Cell {
    int t, i, j, k;
    bool ok;
};

__device__ __forceinline__ Cell tile_cell(const TileItem& ti, int n, int lt, int m) {
    Cell c;
    c.i = ti.i0 + m;
    c.j = ti.j0 + (lt >> 5);
    c.k = ti.k0 + (lt & 31);
    c.ok = c.i < n && c.j < n && c.k < n;
    c.t = (c.i * n + c.j) * n + c.k;
    return c;
}

// Units of a scene's inner products: the scene's T tiles in min(T, kUnits) contiguous runs of nearly equal length.  The
// tile partials of a unit are added in tile order, and the units' sums in a fixed tree over 256 threads (unit u in
// thread u, warp butterfly, warps in order).  Scenes of more than kUnits * kBrickWideTiles tiles are summed without units
// (scene_sums, hf_cg.cu).  The runs depend on the scene alone, so every variant, launch shape and
// batch gives a scene the same bits, and a kernel whose blocks own whole units exchanges one value per unit.
constexpr int kUnits = 148;

__host__ __device__ inline int unit_count(int tiles) { return tiles < kUnits ? tiles : kUnits; }
// (32-bit arithmetic: units are formed of at most kUnits * kBrickWideTiles tiles)
__host__ __device__ inline int unit_first(int tiles, int units, int u) { return tiles * u / units; }

// Per-block copy of a scene's CG scalars; every block derives them from the same partial sums, so all copies agree.
struct LocalScene {
    double rz, atol_sq, bb, rr, pAp, mean;
    double true_rr;             // fp64 |b - A x|^2 of the outer defect correction (-1: not formed)
    float alpha, beta;
    int live, iters, maxit, status;
    int kbase;                  // iterations before the last restart by the defect correction
    int corrections;            // restarts so far
    int dc;                     // the true residual is still to be checked (HF_FLAG_DEFECT_CORRECTION)
};

__device__ __forceinline__ void init_scalars(LocalScene& L, const hf_scene& S, bool heat, const double (&tot)[3], int N) {
    const double tol = heat ? S.heat_tol : S.cg_tol;
    double atol = tol * sqrt(tot[0]);
    if (atol < tol) atol = tol;
    if (atol < 1.0e-18) atol = 1.0e-18;
    int maxit = heat ? S.heat_maxiter : S.cg_max_iter;
    if (maxit <= 0) maxit = N;
    L.maxit = maxit + (maxit & 1);   // iterations run in pairs
    L.bb = tot[0];
    L.rr = tot[1];
    L.rz = tot[2];
    L.atol_sq = atol * atol;
    L.iters = 0;
    L.beta = 0.0f;
    L.alpha = 0.0f;
    L.status = isfinite(tot[1]) ? 0 : HF_SCENE_NONFINITE;
    L.live = tot[1] > L.atol_sq && isfinite(tot[1]) && L.maxit > 0;
    L.true_rr = -1.0;
    L.kbase = 0;
    L.corrections = 0;
    L.dc = (S.flags & HF_FLAG_DEFECT_CORRECTION) != 0;
}

// convergence test after phase B of iteration kit (warp: kernel_2 then the residual test)
__device__ __forceinline__ bool update_scalars(LocalScene& L, bool heat, double rr, double rz, int kit) {
    L.iters = kit;
    const bool above = rr > L.atol_sq;
    L.beta = above ? __double2float_rn(rz / L.rz) : 0.0f;
    L.rz = rz;
    L.rr = rr;
    if (!isfinite(rr)) L.status |= HF_SCENE_NONFINITE;
    const bool live = above && isfinite(rr) && kit < L.maxit;
    if (!live && above && isfinite(rr)) L.status |= heat ? HF_SCENE_HEAT_MAXITER : HF_SCENE_PRESSURE_MAXITER;
    L.live = live;
    return live;
}

__device__ __forceinline__ void write_stats(const hf_scene& S, const LocalScene& L, bool heat, bool timed_out, int par) {
    hf_scene_state* st = S.state;
    if (heat) {
        st->status = L.status | (timed_out ? HF_SCENE_BARRIER_TIMEOUT : 0);
        st->heat_iters = L.iters;
        st->heat_rr = L.rr;
        st->heat_atol = sqrt(L.atol_sq);
        st->heat_bb = L.bb;
        st->heat_true_rr = L.true_rr;
        st->total_heat_iters += L.iters;
    } else {
        st->status |= L.status | (timed_out ? HF_SCENE_BARRIER_TIMEOUT : 0);
        st->pressure_iters = L.iters;
        st->pressure_rr = L.rr;
        st->pressure_atol = sqrt(L.atol_sq);
        st->pressure_bb = L.bb;
        st->pressure_true_rr = L.true_rr;
        st->rhs_mean = L.mean;
        st->total_pressure_iters += L.iters;
        // a substep whose heat solve gave up is not counted either (the heat solve starts the status word anew)
        if (!(st->status & HF_SCENE_BARRIER_TIMEOUT)) {
            st->parity = par ^ 1;
            st->substeps += 1;
        }
    }
}

}  // namespace hf
