// hf_cg.cu -- persistent, cooperative Jacobi-preconditioned CG for the heat and pressure systems of a batch of scenes.
//
// One launch performs a whole solve (heat.py:198-210 or grid.py:235-251) with the convergence test on the device, so
// no iteration waits for the host.  The grid is co-resident (cooperative launch); phases are separated by a software
// grid barrier whose wait is bounded in time (a timeout sets a flag and every block leaves the solve).
//
// Semantics follow warp.optim.linear.cg with M = diag(D) (warp-lang, a dependency of the reference; restated from its
// published algorithm):
//     r = b - A x,  z = D r,  p = z,  atol = max(tol ||b||, tol, 1e-18)
//     repeat: Ap = A p; alpha = rz / pAp; x += alpha p; r -= alpha Ap; z = D r; beta = rz'/rz; p = z + beta p
//     until r.r <= atol^2 (tested every iteration, which is where the reference's frozen iterations leave x) or maxiter.
// Inner products, alpha and beta are fp64; the vectors stay binary32 and alpha/beta are applied after rounding.
//
// Work items are 4 x 8 x 32-cell tiles (i, j, k).  Thread lt of a tile owns cells (i0 + m, j0 + lt/32, k0 + lt%32),
// m = 0..3, so a warp covers one 128-byte k-row.  Each tile yields one fp64 partial per inner product in a fixed tree
// (4 cells in order, warp butterfly, 8 warps in order); a scene's inner product sums its tile partials in tile order
// (again a fixed tree).  Results therefore depend only on the scene -- not on the batch, the grid size or the variant.
//
// Two grid barriers per iteration: the search direction p_k = z + beta p_{k-1} is not a separate phase -- every block
// recomputes it at the stencil points it reads from z and the previous p (double-buffered), so it costs no barrier.
//
// k_pcg streams: the vectors stay in global memory, for any number of scenes of any size (the on-chip solves of hf_brick.cu
// take the plans whose scenes fit there).  The scenes come in L2-sized groups solved by the lanes of the grid; for the
// pressure system with every scene at n % 4 == 0 each tile's stencil boxes and CG vectors are staged by TMA from
// per-scene descriptors, double-buffered per block.  Optional outer defect correction (fp64 true residual, restart).
#include <cuda.h>

#include "hf_cg.cuh"

namespace hf {

// k_pcg's `red` holds kRedComps x 32 doubles: up to 9 components of one sum, or the 8 warps' sums of the group_sums of 36
// scenes and one component.
constexpr int kRedComps = 9;
constexpr int kPlaces = 64;          // tiles of a block whose partials' places a solve keeps (those of more are found each time)
constexpr int kMaxCorrections = 2;   // restarts of one solve by the outer defect correction

// Barrier of nblocks blocks (the grid, or one lane of it) with a bounded wait.  Thread 0 publishes the block's writes with a release reduction (cumulative over
// the writes the block's threads made before __syncthreads) and polls with acquire loads.  Returns false (in every
// thread) once any block has timed out.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned& epoch, int* err, unsigned nblocks) {
    ++epoch;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = epoch * nblocks;
        if (!(epoch == 1 && (int)blockIdx.x == c_absent_block))
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        const unsigned long long t0 = global_timer_ns(), limit = c_wait_limit_ns;
        unsigned spins = 0;
        while (ld_acquire_u32(bar) < target) {
            if (*(volatile int*)err) break;
            if ((++spins & 255u) == 0 && global_timer_ns() - t0 > limit) {
                atomicExch(err, 1);
                break;
            }
        }
    }
    __syncthreads();
    return *(volatile int*)err == 0;
}

// Sum of a scene's partials (item c, component comp[q] at buf[comp[q] * cs + c]: component-major) in a fixed tree: every
// one of the first 256 threads adds its items in order, warp butterfly, then 8 warps in order.  Every block computing it
// obtains the same bits.  Tile partials (cs: the plan's tile count): thread u adds the tiles of unit u (unit_first) when
// the scene is one that the on-chip solve takes; of a larger scene (whose runs of 16 tiles and more would be as many
// dependent round trips), and of the per-chunk rhs sums (cs = 0, one component), thread t adds items t, t + 256, ...
//
// A unit's partials are stored where its thread's loads are coalesced with its neighbours' (part_at): partial q of unit u at
// q * units + u, the last ones of the longer units behind these.  Read from the unit's own run of tiles, every sector was
// fetched up to four times.  us per iteration with the defect correction (whole substep), strided sums / runs / now: 75^3
// 20.2 / 21.4 / 20.8, 96^3 20.1 / 20.7 / 20.1, 128^3 36.4 / 39.8 / 37.6, 160^3 71.8 / 81.5 / 74.4, 168^3 96.1 / 105.1 / 96.0;
// ms per substep of 40 scenes of 48^3 18.9 / 20.1 / 18.4.
struct Run {
    int first, step, count, last;   // items first, first + step, ...; the last one (count - 1) at `last`
    __device__ __forceinline__ int at(int q) const { return q < count - 1 ? first + q * step : last; }
};

// (Of up to kUnits tiles every unit is one: the strided sum is the same.)
__device__ __forceinline__ bool in_units(int T) { return T > kUnits && T <= kUnits * kBrickWideTiles; }

// first tile of unit u of such a scene: unit_first(T, kUnits, u) with a constant divisor (a division by a variable costs 150
// cycles, four times an iteration)
__device__ __forceinline__ int unit_start(int T, int u) { return T * u / kUnits; }

// the items of [b, e) that this thread adds
__device__ __forceinline__ Run thread_run(int b, int e, int cs) {
    const int t = threadIdx.x, T = e - b;
    if (cs == 0 || !in_units(T)) {
        const int count = t < kThreads && t < T ? (T - t + kThreads - 1) / kThreads : 0;
        return Run{b + t, kThreads, count, b + t + (count - 1) * kThreads};
    }
    if (t >= kUnits) return Run{b, 0, 0, b};
    const int least = T / kUnits, first = unit_start(T, t), count = unit_start(T, t + 1) - first;
    return Run{b + t, kUnits, count, b + (count > least ? least * kUnits + first - t * least : t + (least - 1) * kUnits)};
}

// Where the partials of tile c of a scene are kept.  Some 300 cycles for one thread, so a solve finds its tiles' places once
// (kPlaces; in global memory their loads took 6 us an iteration at 180^3).
__device__ __forceinline__ int part_at(const int* __restrict__ tile_begin, int scene, int c) {
    const int b = tile_begin[scene], T = tile_begin[scene + 1] - b, i = c - b;
    if (!in_units(T)) return c;
    int u = (int)(__fdividef((float)(i * kUnits), (float)T));   // within one of the unit that holds i
    u -= unit_start(T, u) > i;
    u += unit_start(T, u + 1) <= i;
    const int first = unit_start(T, u), q = i - first, least = T / kUnits;
    return b + (q < least ? q * kUnits + u : least * kUnits + first - u * least);
}

template <int K, int U = 4>
__device__ __forceinline__ void scene_sums(const double* __restrict__ buf, int b, int e, const int (&comp)[K],
                                           double (&tot)[K], double* red, int cs) {
    static_assert(K <= kRedComps, "red holds kRedComps components");
#pragma unroll
    for (int q = 0; q < K; ++q) tot[q] = 0.0;
    const Run run = thread_run(b, e, cs);
    {
        // U items at a time are loaded (an absent one as +0.0, which leaves a sum that started at +0.0 unchanged) before
        // they are added, so their L2 round trips overlap instead of each waiting for the previous addition
        for (int c = 0; c < run.count; c += U) {
            double v[U][K];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < K; ++q) v[u][q] = c + u < run.count ? buf[comp[q] * cs + run.at(c + u)] : 0.0;
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < K; ++q) tot[q] += v[u][q];
        }
    }
#pragma unroll
    for (int c = 0; c < K; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tot[c] += __shfl_xor_sync(0xffffffffu, tot[c], o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0 && warp < kThreads / 32) {
#pragma unroll
        for (int c = 0; c < K; ++c) red[c * 32 + warp] = tot[c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < K; ++c) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < kThreads / 32; ++q) s += red[c * 32 + q];
        tot[c] = s;
    }
}

// scene_sums for every live scene q < ns of a group (scene scene_lo + q: items tile_begin[s] .. tile_begin[s + 1]), with
// the same tree per scene, in passes of kRedComps * 32 / (8 K) scenes that share one pair of block barriers instead of
// a pair per scene; fn(q, tot) then runs once per live scene, in one thread, with the scene's K sums.  live(q) must
// not change before fn runs for q.  256-thread blocks.
template <int K, class Live, class Fn>
__device__ __forceinline__ void group_sums(const double* __restrict__ buf, const int* __restrict__ tile_begin,
                                           int scene_lo, int ns, const int (&comp)[K], int cs, double* red, Live live,
                                           Fn fn) {
    constexpr int CH = kRedComps * 32 / (8 * K);
    const int lt = threadIdx.x, lane = lt & 31, warp = lt >> 5;
    for (int q0 = 0; q0 < ns; q0 += CH) {
        const int qn = ns - q0 < CH ? ns - q0 : CH;
        for (int qq = 0; qq < qn; ++qq) {
            if (!live(q0 + qq)) continue;
            const int b = tile_begin[scene_lo + q0 + qq], e = tile_begin[scene_lo + q0 + qq + 1];
            double acc[K];
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] = 0.0;
            if (e - b <= kUnits) {   // one item a thread: small scenes in numbers spend their time here
                if (b + lt < e)
#pragma unroll
                    for (int k = 0; k < K; ++k) acc[k] = buf[comp[k] * cs + b + lt];
            } else {
                const Run run = thread_run(b, e, cs);
                constexpr int U = K == 1 ? 14 : 8;   // in flight: as many as fit the registers (14 pairs spill, 39.0 us at 128^3)
                for (int c = 0; c < run.count; c += U) {
                    double v[U][K];
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int k = 0; k < K; ++k) v[u][k] = c + u < run.count ? buf[comp[k] * cs + run.at(c + u)] : 0.0;
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int k = 0; k < K; ++k) acc[k] += v[u][k];
                }
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int k = 0; k < K; ++k) red[(qq * K + k) * 8 + warp] = acc[k];
            }
        }
        __syncthreads();
        if (lt < qn && live(q0 + lt)) {
            double tot[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                double t = 0.0;
#pragma unroll
                for (int w = 0; w < kThreads / 32; ++w) t += red[(lt * K + k) * 8 + w];
                tot[k] = t;
            }
            fn(q0 + lt, tot);
        }
        __syncthreads();
    }
}

// Per-256-thread-group sum (each group reduces its own 8 warps in index order): the tile partial tree.
template <int K>
__device__ __forceinline__ void group_sum(double (&v)[K], double* red) {
    static_assert(K <= kRedComps, "red holds kRedComps components");
#pragma unroll
    for (int c = 0; c < K; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g0 = (warp >> 3) << 3;
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < K; ++c) red[c * 32 + warp] = v[c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < K; ++c) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += red[c * 32 + g0 + q];
        v[c] = s;
    }
}

// Search direction at cell t for iteration k: p_k = z + beta p_{k-1} (warp's _cg_kernel_2), or z at k = 1.
struct Dir {
    const float* z;
    const float* pold;
    float beta;
    bool first;
    __device__ __forceinline__ float operator()(int t) const {
        return first ? z[t] : __fadd_rn(z[t], __fmul_rn(beta, pold[t]));
    }
};

// grid.py:94-115 k_laplacian accumulation, the sum over the six faces of alpha_f (x_c - x_nb) with domain faces skipped,
// every load hoisted: each is in bounds (a missing neighbour reads the cell itself, face fractions exist on all n+1
// layers), so all of a thread's loads are in flight at once; the terms of domain faces are then left out of the sum, in
// the reference's order.
template <class X>
__device__ __forceinline__ float lap_acc_hoisted(const hf_scene& S, const X& x, float xc, int t, int i, int j, int k) {
    const int n = S.n, nn = n * n;
    const bool in0 = i > 0, in1 = i < n - 1, in2 = j > 0, in3 = j < n - 1, in4 = k > 0, in5 = k < n - 1;
    const float x0 = x(in0 ? t - nn : t), x1 = x(in1 ? t + nn : t), x2 = x(in2 ? t - n : t), x3 = x(in3 ? t + n : t),
                x4 = x(in4 ? t - 1 : t), x5 = x(in5 ? t + 1 : t);
    const float a0 = __ldg(S.ax + uidx_(n, i, j, k)), a1 = __ldg(S.ax + uidx_(n, i + 1, j, k)),
                a2 = __ldg(S.ay + vidx_(n, i, j, k)), a3 = __ldg(S.ay + vidx_(n, i, j + 1, k)),
                a4 = __ldg(S.az + widx_(n, i, j, k)), a5 = __ldg(S.az + widx_(n, i, j, k + 1));
    float acc = 0.0f;
    if (in0) acc = __fadd_rn(acc, __fmul_rn(a0, __fsub_rn(xc, x0)));
    if (in1) acc = __fadd_rn(acc, __fmul_rn(a1, __fsub_rn(xc, x1)));
    if (in2) acc = __fadd_rn(acc, __fmul_rn(a2, __fsub_rn(xc, x2)));
    if (in3) acc = __fadd_rn(acc, __fmul_rn(a3, __fsub_rn(xc, x3)));
    if (in4) acc = __fadd_rn(acc, __fmul_rn(a4, __fsub_rn(xc, x4)));
    if (in5) acc = __fadd_rn(acc, __fmul_rn(a5, __fsub_rn(xc, x5)));
    return acc;
}

// heat.py:55-91 neighbour_terms with use_fixed = 0; kappa_f from the precomputed face diffusivities (loads hoisted
// and kept in bounds as in lap_acc_hoisted)
template <class X>
__device__ __forceinline__ float heat_nt_hoisted(const hf_scene& S, const X& x, float xc, int t, int i, int j, int k) {
    const int n = S.n, nn = n * n;
    const uint8_t* __restrict__ fl = S.cell_flags;
    const bool in[6] = {i > 0, i < n - 1, j > 0, j < n - 1, k > 0, k < n - 1};
    const int step[6] = {-nn, nn, -n, n, -1, 1};
    const int fidx[6] = {uidx_(n, i, j, k), uidx_(n, i + 1, j, k), vidx_(n, i, j, k), vidx_(n, i, j + 1, k),
                         widx_(n, i, j, k), widx_(n, i, j, k + 1)};
    const float* __restrict__ hk[3] = {S.hkx, S.hky, S.hkz};
    float xn[6], kf[6];
    uint8_t fn[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        const int nb = in[s] ? t + step[s] : t;
        xn[s] = x(nb);
        fn[s] = __ldg(fl + nb);
        kf[s] = __ldg(hk[s >> 1] + fidx[s]);
    }
    float acc = 0.0f;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        if (!in[s]) continue;
        acc = __fadd_rn(acc, (fn[s] & 1) ? __fmul_rn(kf[s], xc) : __fmul_rn(kf[s], __fsub_rn(xc, xn[s])));
    }
    return acc;
}

// Set-up of one cell (heat.py:198-203 + k_heat_rhs/k_heat_diag; grid.py:238-248 mean removal + k_jacobi): returns
// b, D, r for x0 (the advected T, or the previous pressure).  Every load comes first and stays in bounds (a missing
// neighbour reads the cell itself), so they are in flight together; the sums then take the in-domain terms in the
// reference's order (heat.py:121-144 k_heat_diag and heat_nt, or k_jacobi's face-fraction sum and lap_acc).
template <bool HEAT>
__device__ __forceinline__ void setup_cell(const hf_scene& S, const float* x, float mean, float hh, float c_dt,
                                           const Cell& c, float& b, float& d, float& r) {
    const int n = S.n, nn = n * n, t = c.t, i = c.i, j = c.j, k = c.k;
    const bool in[6] = {i > 0, i < n - 1, j > 0, j < n - 1, k > 0, k < n - 1};
    const int step[6] = {-nn, nn, -n, n, -1, 1};
    const int fidx[6] = {uidx_(n, i, j, k), uidx_(n, i + 1, j, k), vidx_(n, i, j, k), vidx_(n, i, j + 1, k),
                         widx_(n, i, j, k), widx_(n, i, j, k + 1)};
    const float xc = x[t];
    float xn[6], kf[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) xn[s] = x[in[s] ? t + step[s] : t];
    if (HEAT) {
        const float* __restrict__ hk[3] = {S.hkx, S.hky, S.hkz};
        const uint8_t* __restrict__ fl = S.cell_flags;
        uint8_t fn[6];
#pragma unroll
        for (int s = 0; s < 6; ++s) {
            kf[s] = __ldg(hk[s >> 1] + fidx[s]);
            fn[s] = __ldg(fl + (in[s] ? t + step[s] : t));
        }
        b = S.hrhs[t];
        if (fl[t] & 1) {
            d = 1.0f;
            r = __fsub_rn(b, xc);
        } else {
            float sd = 0.0f, nt = 0.0f;
#pragma unroll
            for (int s = 0; s < 6; ++s)
                if (in[s]) sd = __fadd_rn(sd, kf[s]);
#pragma unroll
            for (int s = 0; s < 6; ++s) {
                if (!in[s]) continue;
                nt = __fadd_rn(nt, (fn[s] & 1) ? __fmul_rn(kf[s], xc) : __fmul_rn(kf[s], __fsub_rn(xc, xn[s])));
            }
            d = __fdiv_rn(1.0f, __fadd_rn(1.0f, __fmul_rn(c_dt, sd)));
            r = __fsub_rn(b, __fadd_rn(xc, __fmul_rn(c_dt, nt)));
        }
    } else {
        const float* __restrict__ af[3] = {S.ax, S.ay, S.az};
#pragma unroll
        for (int s = 0; s < 6; ++s) kf[s] = __ldg(af[s >> 1] + fidx[s]);
        b = S.rhs[t];
        if (mean != 0.0f) {
            b = __fsub_rn(b, mean);
            S.rhs[t] = b;
        }
        float sa = 0.0f, acc = 0.0f;
#pragma unroll
        for (int s = 0; s < 6; ++s)
            if (in[s]) sa = __fadd_rn(sa, kf[s]);
#pragma unroll
        for (int s = 0; s < 6; ++s)
            if (in[s]) acc = __fadd_rn(acc, __fmul_rn(kf[s], __fsub_rn(xc, xn[s])));
        d = __fdiv_rn(hh, maxf_(sa, 1.0e-12f));
        r = __fsub_rn(b, __fdiv_rn(acc, hh));
    }
}

// grid.py:140-153 k_project for the three low faces of a cell (and the high wall faces on the last layer)
__device__ __forceinline__ void project_cell(const hf_scene& S, float* u, float* v, float* w, const float* p, float pc,
                                             float dtr, float h, const Cell& c) {
    const int n = S.n, nn = n * n, t = c.t, i = c.i, j = c.j, k = c.k;
    int f = uidx_(n, i, j, k);
    u[f] = i == 0 ? 0.0f : __fsub_rn(u[f], __fdiv_rn(__fmul_rn(dtr, __fsub_rn(pc, p[t - nn])), h));
    f = vidx_(n, i, j, k);
    v[f] = j == 0 ? 0.0f : __fsub_rn(v[f], __fdiv_rn(__fmul_rn(dtr, __fsub_rn(pc, p[t - n])), h));
    f = widx_(n, i, j, k);
    w[f] = k == 0 ? 0.0f : __fsub_rn(w[f], __fdiv_rn(__fmul_rn(dtr, __fsub_rn(pc, p[t - 1])), h));
    if (i == n - 1) u[uidx_(n, n, j, k)] = 0.0f;
    if (j == n - 1) v[vidx_(n, i, n, k)] = 0.0f;
    if (k == n - 1) w[widx_(n, i, j, n)] = 0.0f;
}

// True residual b - A x of one cell for the outer defect correction: the binary32 operator (grid.py:94-115 with the
// binary32 h^2; heat.py:94-105 with the binary32 dt/h^2 and face diffusivities) applied with every product and sum in
// fp64 to the binary32 vectors.
__device__ double true_residual_pressure(const hf_scene& S, const float* __restrict__ x, int t, int i, int j, int k,
                                         double hh) {
    const int n = S.n, nn = n * n;
    const double xc = x[t];
    double acc = 0.0;
    if (i > 0) acc += (double)S.ax[uidx_(n, i, j, k)] * (xc - (double)x[t - nn]);
    if (i < n - 1) acc += (double)S.ax[uidx_(n, i + 1, j, k)] * (xc - (double)x[t + nn]);
    if (j > 0) acc += (double)S.ay[vidx_(n, i, j, k)] * (xc - (double)x[t - n]);
    if (j < n - 1) acc += (double)S.ay[vidx_(n, i, j + 1, k)] * (xc - (double)x[t + n]);
    if (k > 0) acc += (double)S.az[widx_(n, i, j, k)] * (xc - (double)x[t - 1]);
    if (k < n - 1) acc += (double)S.az[widx_(n, i, j, k + 1)] * (xc - (double)x[t + 1]);
    return (double)S.rhs[t] - acc / hh;
}

__device__ double true_residual_heat(const hf_scene& S, const float* __restrict__ x, int t, int i, int j, int k,
                                     double c_dt) {
    const int n = S.n, nn = n * n;
    const double xc = x[t], b = S.hrhs[t];
    if (S.cell_flags[t] & 1) return b - xc;
    const int nbr[6] = {t - nn, t + nn, t - n, t + n, t - 1, t + 1};
    const bool in[6] = {i > 0, i < n - 1, j > 0, j < n - 1, k > 0, k < n - 1};
    const int fidx[6] = {uidx_(n, i, j, k), uidx_(n, i + 1, j, k), vidx_(n, i, j, k), vidx_(n, i, j + 1, k),
                         widx_(n, i, j, k), widx_(n, i, j, k + 1)};
    const float* hk[3] = {S.hkx, S.hky, S.hkz};
    double acc = 0.0;
    for (int q = 0; q < 6; ++q) {
        if (!in[q]) continue;
        const double kf = hk[q >> 1][fidx[q]];
        acc += (S.cell_flags[nbr[q]] & 1) ? kf * xc : kf * (xc - (double)x[nbr[q]]);
    }
    return b - (xc + c_dt * acc);
}

// ============================================================================================ TMA staging
// Box geometry of the tiled pressure stencil (elements, innermost k first), all at 16-byte aligned k origins:
//   z / p_old : k in [k0-4, k0+36), j in [j0-1, j0+9), i in [i0-1, i0+5)   (one-cell halo; k widened to alignment)
//   alpha_f x : k in [k0, k0+32),   j in [j0, j0+8),   i in [i0, i0+5)     (low faces of the tile + next i layer)
//   alpha_f y : k in [k0, k0+32),   j in [j0, j0+9),   i in [i0, i0+4)
//   alpha_f z : k in [k0, k0+36),   j in [j0, j0+8),   i in [i0, i0+4)
// Out-of-range elements are zero-filled by the copy engine and never used (domain faces are skipped).
constexpr int kBZ = 40 * 10 * 6, kBX = 32 * 8 * 5, kBY = 32 * 9 * 4, kBW = 36 * 8 * 4;
constexpr int kSlotFloats = 2 * kBZ + kBX + kBY + kBW;   // 8384 floats = 33,536 bytes (a multiple of 128)

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// The first 128-byte aligned float of the dynamic shared memory (TMA destinations), derived from raw by pointer
// arithmetic so that the compiler keeps the shared address space: a round trip through an integer would turn every
// access to the boxes into a generic load or store.
__device__ __forceinline__ float* align128_shared(float* raw) {
    return raw + ((128u - (smem_addr(raw) & 127u)) & 127u) / 4u;
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

// bounded wait for the given phase; returns false on timeout
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned phase) {
    const unsigned long long t0 = global_timer_ns();
    for (unsigned spins = 0;; ++spins) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(phase)
            : "memory");
        if (ok) return true;
        if ((spins & 63u) == 63u && global_timer_ns() - t0 > c_wait_limit_ns) return false;
    }
}

__device__ __forceinline__ void tma_load_3d(float* dst, const CUtensorMap* map, int x, int y, int z, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

// Tiles c = first, first + step, ... < end of scenes still iterating, through two shared-memory slots: the boxes of the
// next tile are requested (issue, thread 0) before the current tile is worked on, so the copy overlaps the work.  Bit s
// of ph is the phase the next wait on slot s expects.
// `work` must end with a __syncthreads after its last read of the slot (the slot is refilled next).  A wait that times
// out sets the error flag and waits once more for the copy, so that no copy is left in flight.
template <class Issue, class Work>
__device__ __forceinline__ void pipelined_tiles(int first, int end, int step, const LocalScene* loc, int scene_lo,
                                                const TileItem* __restrict__ tiles, float* slots,
                                                unsigned long long* mbar, unsigned& ph, int* err, Issue issue, Work work) {
    auto next_live = [&](int c, int& nth) {
        while (c < end && !loc[tiles[c].scene - scene_lo].live) c += step, ++nth;
        return c;
    };
    int nth = 0, si = 0, cur = next_live(first, nth);
    if (cur < end && threadIdx.x == 0) issue(cur, slots, &mbar[0]);
    while (cur < end) {
        int nth_nxt = nth + 1;
        const int nxt = next_live(cur + step, nth_nxt);
        if (nxt < end && threadIdx.x == 0) issue(nxt, slots + (si ^ 1) * kSlotFloats, &mbar[si ^ 1]);
        const unsigned phase = (ph >> si) & 1u;
        if (!mbar_wait(&mbar[si], phase)) {
            if (threadIdx.x == 0) atomicExch(err, 1);
            mbar_wait(&mbar[si], phase);
        }
        ph ^= 1u << si;
        work(cur, slots + si * kSlotFloats, nth);
        cur = nxt;
        nth = nth_nxt;
        si ^= 1;
    }
}

// ================================================================================================== streaming
// A launch solves the groups of a GroupTable: consecutive scenes whose CG vectors the host sized to stay in L2.  The
// grid is split into gt.lanes lanes of equal size (lane = blockIdx.x / blocks per lane), each with its own barrier;
// a lane takes the next unsolved group from a queue counter, so independent groups run side by side and one lane's
// barrier waits overlap another lane's stencils on the same SM.  Inside a group, tiles are dealt round-robin over the
// lane's blocks (an equal share of every live scene per block while scenes converge at different iterations); every
// block sums the tile partials of every scene of the group itself (same bits everywhere) and keeps the scalars in
// shared memory, so an iteration takes two lane barriers.  Returns false when a barrier timed out.
template <bool HEAT, bool TMA>
__device__ bool solve_group(const hf_scene* __restrict__ scenes, const TileItem* __restrict__ tiles, const int4 grp,
                            int lb, int nlb, unsigned* bar, unsigned& epoch, double dt_d, const Workspace& ws,
                            double* red, LocalScene* loc, unsigned char* s_par, int* s_any, float* slots,
                            unsigned long long* mbar, unsigned& ph, int* place) {
    const int scene_lo = grp.x, scene_hi = grp.y, tile_lo = grp.z, tile_hi = grp.w;
    const int ns = scene_hi - scene_lo;
    double* bufA = ws.partA;
    double* bufB = ws.partB;
    // part_at of this block's nth tile (thread 0)
    auto placed = [&](int nth, int scene, int c) { return nth < kPlaces ? place[nth] : part_at(ws.tile_begin, scene, c); };
    const float dt = (float)dt_d;
    const int lt = threadIdx.x;
    const int first = tile_lo + lb;
    bool ok = true;
    if (threadIdx.x < ns) s_par[threadIdx.x] = (unsigned char)scenes[scene_lo + threadIdx.x].state->parity;

    // ---------------------------------------------------------------------------------------- prologue
    for (int q = 0; q < ns; ++q) {
        const int s = scene_lo + q;
        if (!HEAT) {
            // the pressure rhs mean (grid.py:238-241) from the divergence stage's chunk sums
            double m[1];
            const int comp[1] = {0};
            scene_sums<1>(ws.mean_part, ws.chunk_begin[s], ws.chunk_begin[s + 1], comp, m, red, 0);
            const int n = scenes[s].n;
            if (threadIdx.x == 0) loc[q].mean = (double)__double2float_rn(m[0] / ((double)n * n * n));
        } else if (threadIdx.x == 0) {
            loc[q].mean = 0.0;
        }
    }
    __syncthreads();
    for (int c = first, nth = 0; c < tile_hi; c += nlb, ++nth) {
        const TileItem ti = tiles[c];
        const hf_scene& S = scenes[ti.scene];
        const int n = S.n, par = s_par[ti.scene - scene_lo];
        const float h = (float)S.h, hh = __fmul_rn(h, h), c_dt = __fdiv_rn(dt, hh);
        const float* x = HEAT ? S.T[par ^ 1] : S.p;
        const float mean = (float)loc[ti.scene - scene_lo].mean;
        double part[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const Cell cl = tile_cell(ti, n, lt, m);
            if (!cl.ok) continue;
            float b, d, r;
            setup_cell<HEAT>(S, x, mean, hh, c_dt, cl, b, d, r);
            const float z = __fmul_rn(d, r);
            (HEAT ? S.hdiag : S.pdiag)[cl.t] = d;
            S.cg_r[cl.t] = r;
            S.cg_z[cl.t] = z;
            part[0] += (double)b * (double)b;
            part[1] += (double)r * (double)r;
            part[2] += (double)r * (double)z;
        }
        group_sum<3>(part, red);
        if (lt == 0) {
            const int at = part_at(ws.tile_begin, ti.scene, c);
            if (nth < kPlaces) place[nth] = at;
            bufB[at] = part[0];
            bufB[1 * ws.tiles + at] = part[1];
            bufB[2 * ws.tiles + at] = part[2];
        }
    }
    if (!(ok = grid_barrier(bar, epoch, ws.err, nlb))) goto done;
    for (int q = 0; q < ns; ++q) {
        const int s = scene_lo + q;
        const int b = ws.tile_begin[s], e = ws.tile_begin[s + 1];
        double tot[3];
        const int comp[3] = {0, 1, 2};
        scene_sums<3>(bufB, b, e, comp, tot, red, ws.tiles);
        if (threadIdx.x == 0) {
            const hf_scene& S = scenes[s];
            const double mean = loc[q].mean;
            init_scalars(loc[q], S, HEAT, tot, S.n * S.n * S.n);
            loc[q].mean = mean;
            loc[q].live = loc[q].live && b < e;
        }
    }
    if (threadIdx.x == 0) {
        int any = 0;
        for (int q = 0; q < ns; ++q) any |= loc[q].live;
        *s_any = any;
    }
    __syncthreads();

    // ------------------------------------------------------------------------------------------ iterations
    // Rounds: CG iterations until every scene has stopped; then, for scenes with the outer defect correction, the true
    // residual, and another round for the scenes it restarted.
    for (;;) {
    for (int kit = 1; *s_any; ++kit) {
        // phase A: p_k at the stencil points, Ap = A p_k, p.Ap
        if constexpr (TMA) {
            // stage z and p_{k-1} with a one-cell halo and the tile's face fractions, form p_k in place, A p from shared memory
            const bool first_it = kit == 1;
            auto issue = [&](int c, float* slot, unsigned long long* mb) {
                const TileItem ti = tiles[c];
                asm volatile("fence.proxy.async.global;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                const bool go = *(volatile int*)ws.err == 0;
                const CUtensorMap* M = ws.maps + kMapsPerScene * ti.scene;
                mbar_expect_tx(mb, go ? (unsigned)(((first_it ? 1 : 2) * kBZ + kBX + kBY + kBW) * sizeof(float)) : 0u);
                if (go) {
                    tma_load_3d(slot, &M[0], ti.k0 - 4, ti.j0 - 1, ti.i0 - 1, mb);
                    if (!first_it) tma_load_3d(slot + kBZ, &M[1 + ((kit - 1) & 1)], ti.k0 - 4, ti.j0 - 1, ti.i0 - 1, mb);
                    tma_load_3d(slot + 2 * kBZ, &M[3], ti.k0, ti.j0, ti.i0, mb);
                    tma_load_3d(slot + 2 * kBZ + kBX, &M[4], ti.k0, ti.j0, ti.i0, mb);
                    tma_load_3d(slot + 2 * kBZ + kBX + kBY, &M[5], ti.k0, ti.j0, ti.i0, mb);
                }
            };
            auto work = [&](int c, float* slot, int nth) {
                const TileItem ti = tiles[c];
                const LocalScene& L = loc[ti.scene - scene_lo];
                const hf_scene& S = scenes[ti.scene];
                const int n = S.n;
                const float h = (float)S.h, hh = __fmul_rn(h, h);
                if (!first_it)
                    for (int e = lt; e < kBZ; e += kThreads) slot[e] = __fadd_rn(slot[e], __fmul_rn(L.beta, slot[kBZ + e]));
                __syncthreads();
                const float* axb = slot + 2 * kBZ;
                const float* ayb = axb + kBX;
                const float* azb = ayb + kBY;
                float* pnew = S.cg_p[kit & 1];
                double part[1] = {0.0};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const Cell cl = tile_cell(ti, n, lt, m);
                    if (!cl.ok) continue;
                    const int bi = m, bj = lt >> 5, bk = lt & 31;
                    const int o = (bi + 1) * 400 + (bj + 1) * 40 + (bk + 4);
                    const float pc = slot[o];
                    float acc = 0.0f;
                    if (cl.i > 0) acc = __fadd_rn(acc, __fmul_rn(axb[bi * 256 + bj * 32 + bk], __fsub_rn(pc, slot[o - 400])));
                    if (cl.i < n - 1)
                        acc = __fadd_rn(acc, __fmul_rn(axb[(bi + 1) * 256 + bj * 32 + bk], __fsub_rn(pc, slot[o + 400])));
                    if (cl.j > 0) acc = __fadd_rn(acc, __fmul_rn(ayb[bi * 288 + bj * 32 + bk], __fsub_rn(pc, slot[o - 40])));
                    if (cl.j < n - 1)
                        acc = __fadd_rn(acc, __fmul_rn(ayb[bi * 288 + (bj + 1) * 32 + bk], __fsub_rn(pc, slot[o + 40])));
                    if (cl.k > 0) acc = __fadd_rn(acc, __fmul_rn(azb[bi * 288 + bj * 36 + bk], __fsub_rn(pc, slot[o - 1])));
                    if (cl.k < n - 1)
                        acc = __fadd_rn(acc, __fmul_rn(azb[bi * 288 + bj * 36 + bk + 1], __fsub_rn(pc, slot[o + 1])));
                    const float ap = __fdiv_rn(acc, hh);
                    pnew[cl.t] = pc;
                    S.cg_Ap[cl.t] = ap;
                    part[0] += (double)pc * (double)ap;
                }
                group_sum<1>(part, red);   // its __syncthreads also ends every read of the slot
                if (lt == 0) bufA[placed(nth, ti.scene, c)] = part[0];
            };
            pipelined_tiles(first, tile_hi, nlb, loc, scene_lo, tiles, slots, mbar, ph, ws.err, issue, work);
        }
        for (int c = first, nth = 0; !TMA && c < tile_hi; c += nlb, ++nth) {
            const TileItem ti = tiles[c];
            const LocalScene& L = loc[ti.scene - scene_lo];
            if (!L.live) continue;
            const hf_scene& S = scenes[ti.scene];
            const int n = S.n;
            const float h = (float)S.h, hh = __fmul_rn(h, h), c_dt = __fdiv_rn(dt, hh);
            const Dir P{S.cg_z, S.cg_p[(kit - 1) & 1], L.beta, kit == 1};
            float pc[4], ap[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const Cell cl = tile_cell(ti, n, lt, m);
                pc[m] = ap[m] = 0.0f;
                if (!cl.ok) continue;
                pc[m] = P(cl.t);
                if (HEAT) {
                    ap[m] = (__ldg(S.cell_flags + cl.t) & 1)
                                ? pc[m]
                                : __fadd_rn(pc[m], __fmul_rn(c_dt, heat_nt_hoisted(S, P, pc[m], cl.t, cl.i, cl.j, cl.k)));
                } else {
                    ap[m] = __fdiv_rn(lap_acc_hoisted(S, P, pc[m], cl.t, cl.i, cl.j, cl.k), hh);
                }
            }
            float* pnew = S.cg_p[kit & 1];
            double part[1] = {0.0};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const Cell cl = tile_cell(ti, n, lt, m);
                if (!cl.ok) continue;
                pnew[cl.t] = pc[m];
                S.cg_Ap[cl.t] = ap[m];
                part[0] += (double)pc[m] * (double)ap[m];
            }
            group_sum<1>(part, red);
            if (lt == 0) bufA[placed(nth, ti.scene, c)] = part[0];
        }
        if (!(ok = grid_barrier(bar, epoch, ws.err, nlb))) goto done;
        {
            // every live scene's p.Ap (live: shared values written before the last __syncthreads)
            const int comp[1] = {0};
            group_sums<1>(bufA, ws.tile_begin, scene_lo, ns, comp, ws.tiles, red, [&](int q) { return (bool)loc[q].live; },
                          [&](int q, const double(&tot)[1]) {
                              loc[q].pAp = tot[0];
                              loc[q].alpha = __double2float_rn(loc[q].rz / tot[0]);
                          });
        }
        // phase B: x += alpha p, r -= alpha Ap, z = D r, r.r and r.z
        if constexpr (TMA) {
            // the tile's x, p_k, r, Ap and D as five (32, 8, 4) boxes: element (m, lt / 32, lt % 32) at m 256 + lt
            auto issue = [&](int c, float* slot, unsigned long long* mb) {
                const TileItem ti = tiles[c];
                asm volatile("fence.proxy.async.global;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                const bool go = *(volatile int*)ws.err == 0;
                const CUtensorMap* M = ws.maps + kMapsPerScene * ti.scene;
                mbar_expect_tx(mb, go ? (unsigned)(5 * 1024 * sizeof(float)) : 0u);
                if (go) {
                    tma_load_3d(slot, &M[6], ti.k0, ti.j0, ti.i0, mb);
                    tma_load_3d(slot + 1024, &M[7 + (kit & 1)], ti.k0, ti.j0, ti.i0, mb);
                    tma_load_3d(slot + 2048, &M[9], ti.k0, ti.j0, ti.i0, mb);
                    tma_load_3d(slot + 3072, &M[10], ti.k0, ti.j0, ti.i0, mb);
                    tma_load_3d(slot + 4096, &M[11], ti.k0, ti.j0, ti.i0, mb);
                }
            };
            auto work = [&](int c, float* slot, int nth) {
                const TileItem ti = tiles[c];
                const LocalScene& L = loc[ti.scene - scene_lo];
                const hf_scene& S = scenes[ti.scene];
                const int n = S.n;
                const float alpha = L.alpha;
                double part[2] = {0.0, 0.0};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const Cell cl = tile_cell(ti, n, lt, m);
                    if (!cl.ok) continue;
                    const int e = m * 256 + lt;
                    const float xv = __fadd_rn(slot[e], __fmul_rn(alpha, slot[1024 + e]));
                    const float rv = __fsub_rn(slot[2048 + e], __fmul_rn(alpha, slot[3072 + e]));
                    const float zv = __fmul_rn(slot[4096 + e], rv);
                    S.p[cl.t] = xv;
                    S.cg_r[cl.t] = rv;
                    S.cg_z[cl.t] = zv;
                    part[0] += (double)rv * (double)rv;
                    part[1] += (double)rv * (double)zv;
                }
                group_sum<2>(part, red);
                if (lt == 0) {
                    const int at = placed(nth, ti.scene, c);
                    bufB[1 * ws.tiles + at] = part[0];
                    bufB[2 * ws.tiles + at] = part[1];
                }
            };
            pipelined_tiles(first, tile_hi, nlb, loc, scene_lo, tiles, slots, mbar, ph, ws.err, issue, work);
        }
        for (int c = first, nth = 0; !TMA && c < tile_hi; c += nlb, ++nth) {
            const TileItem ti = tiles[c];
            const LocalScene& L = loc[ti.scene - scene_lo];
            if (!L.live) continue;
            const hf_scene& S = scenes[ti.scene];
            const int n = S.n, par = s_par[ti.scene - scene_lo];
            float* x = HEAT ? S.T[par ^ 1] : S.p;
            const float* D = HEAT ? S.hdiag : S.pdiag;
            const float* pk = S.cg_p[kit & 1];
            const float alpha = L.alpha;
            float xv[4], rv[4], zv[4];
            {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const Cell cl = tile_cell(ti, n, lt, m);
                    xv[m] = rv[m] = zv[m] = 0.0f;
                    if (!cl.ok) continue;
                    xv[m] = __fadd_rn(x[cl.t], __fmul_rn(alpha, pk[cl.t]));
                    rv[m] = __fsub_rn(S.cg_r[cl.t], __fmul_rn(alpha, S.cg_Ap[cl.t]));
                    zv[m] = __fmul_rn(D[cl.t], rv[m]);
                }
            }
            double part[2] = {0.0, 0.0};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const Cell cl = tile_cell(ti, n, lt, m);
                if (!cl.ok) continue;
                x[cl.t] = xv[m];
                S.cg_r[cl.t] = rv[m];
                S.cg_z[cl.t] = zv[m];
                part[0] += (double)rv[m] * (double)rv[m];
                part[1] += (double)rv[m] * (double)zv[m];
            }
            group_sum<2>(part, red);
            if (lt == 0) {
                const int at = placed(nth, ti.scene, c);
                bufB[1 * ws.tiles + at] = part[0];
                bufB[2 * ws.tiles + at] = part[1];
            }
        }
        if (!(ok = grid_barrier(bar, epoch, ws.err, nlb))) goto done;
        {
            // every live scene's r.r and r.z, then its convergence test
            const int comp[2] = {1, 2};
            group_sums<2>(bufB, ws.tile_begin, scene_lo, ns, comp, ws.tiles, red, [&](int q) { return (bool)loc[q].live; },
                          [&](int q, const double(&tot)[2]) { update_scalars(loc[q], HEAT, tot[0], tot[1], loc[q].kbase + kit); });
        }
        if (threadIdx.x == 0) {
            int any = 0;
            for (int q = 0; q < ns; ++q) any |= loc[q].live;
            *s_any = any;
        }
        __syncthreads();
    }
    // ------------------------------------------------------------- outer defect correction (fp64 true residual)
    if (threadIdx.x == 0) {
        int any = 0;
        for (int q = 0; q < ns; ++q) any |= loc[q].dc;
        *s_any = any;
    }
    __syncthreads();
    if (!*s_any) break;
    // pass 1: r_true = b - A x in fp64 for the scenes to check, rounded into the Ap vector (free between solves)
    for (int c = first; c < tile_hi; c += nlb) {
        const TileItem ti = tiles[c];
        if (!loc[ti.scene - scene_lo].dc) continue;
        const hf_scene& S = scenes[ti.scene];
        const int n = S.n, par = s_par[ti.scene - scene_lo];
        const float h = (float)S.h, hh = __fmul_rn(h, h), c_dt = __fdiv_rn(dt, hh);
        const float* x = HEAT ? S.T[par ^ 1] : S.p;
        double part[1] = {0.0};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const Cell cl = tile_cell(ti, n, lt, m);
            if (!cl.ok) continue;
            const double rt = HEAT ? true_residual_heat(S, x, cl.t, cl.i, cl.j, cl.k, (double)c_dt)
                                   : true_residual_pressure(S, x, cl.t, cl.i, cl.j, cl.k, (double)hh);
            S.cg_Ap[cl.t] = __double2float_rn(rt);
            part[0] += rt * rt;
        }
        group_sum<1>(part, red);
        if (lt == 0) bufA[1 * ws.tiles + part_at(ws.tile_begin, ti.scene, c)] = part[0];
    }
    if (!(ok = grid_barrier(bar, epoch, ws.err, nlb))) goto done;
    for (int q = 0; q < ns; ++q) {
        if (!loc[q].dc) continue;   // uniform: shared value
        const int s = scene_lo + q;
        double tot[1];
        const int comp[1] = {1};
        scene_sums<1>(bufA, ws.tile_begin[s], ws.tile_begin[s + 1], comp, tot, red, ws.tiles);
        if (threadIdx.x == 0) {
            LocalScene& L = loc[q];
            L.true_rr = tot[0];
            // restart from x with the true residual when it is above the tolerance, the recurrence had converged
            // (not stopped at maxiter or on a non-finite value) and corrections are left
            const bool stopped = L.status & (HF_SCENE_NONFINITE | HF_SCENE_HEAT_MAXITER | HF_SCENE_PRESSURE_MAXITER);
            L.live = isfinite(tot[0]) && tot[0] > L.atol_sq && !stopped && L.corrections < kMaxCorrections &&
                     L.iters < L.maxit;
            L.dc = L.live;
            if (L.live) {
                L.corrections += 1;
                L.status |= HF_SCENE_CORRECTED;
                L.kbase = L.iters;
            }
        }
    }
    if (threadIdx.x == 0) {
        int any = 0;
        for (int q = 0; q < ns; ++q) any |= loc[q].live;
        *s_any = any;
    }
    __syncthreads();
    if (!*s_any) break;
    // pass 2: r = r_true, z = D r for the restarted scenes; r.r and r.z start the next round (p_1 = z)
    for (int c = first; c < tile_hi; c += nlb) {
        const TileItem ti = tiles[c];
        if (!loc[ti.scene - scene_lo].live) continue;
        const hf_scene& S = scenes[ti.scene];
        const int n = S.n;
        const float* D = HEAT ? S.hdiag : S.pdiag;
        double part[2] = {0.0, 0.0};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const Cell cl = tile_cell(ti, n, lt, m);
            if (!cl.ok) continue;
            const float r = S.cg_Ap[cl.t];
            const float z = __fmul_rn(D[cl.t], r);
            S.cg_r[cl.t] = r;
            S.cg_z[cl.t] = z;
            part[0] += (double)r * (double)r;
            part[1] += (double)r * (double)z;
        }
        group_sum<2>(part, red);
        if (lt == 0) {
            const int at = part_at(ws.tile_begin, ti.scene, c);
            bufB[1 * ws.tiles + at] = part[0];
            bufB[2 * ws.tiles + at] = part[1];
        }
    }
    if (!(ok = grid_barrier(bar, epoch, ws.err, nlb))) goto done;
    for (int q = 0; q < ns; ++q) {
        if (!loc[q].live) continue;
        const int s = scene_lo + q;
        double tot[2];
        const int comp[2] = {1, 2};
        scene_sums<2>(bufB, ws.tile_begin[s], ws.tile_begin[s + 1], comp, tot, red, ws.tiles);
        if (threadIdx.x == 0) {
            LocalScene& L = loc[q];
            L.rr = tot[0];
            L.rz = tot[1];
            L.beta = 0.0f;
            L.live = isfinite(tot[0]) && tot[0] > L.atol_sq;
        }
    }
    if (threadIdx.x == 0) {
        int any = 0;
        for (int q = 0; q < ns; ++q) any |= loc[q].live;
        *s_any = any;
    }
    __syncthreads();
    }   // rounds
    // -------------------------------------------------------------------- pressure epilogue: projection
    if (!HEAT) {
        for (int c = first; c < tile_hi; c += nlb) {
            const TileItem ti = tiles[c];
            const hf_scene& S = scenes[ti.scene];
            const int n = S.n, par = s_par[ti.scene - scene_lo];
            const float h = (float)S.h, dtr = (float)(dt_d / S.rho);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const Cell cl = tile_cell(ti, n, lt, m);
                if (cl.ok) project_cell(S, S.u[par ^ 1], S.v[par ^ 1], S.w[par ^ 1], S.p, S.p[cl.t], dtr, h, cl);
            }
        }
    }
done:
    // Every block of the lane read the group's parities before its first barrier, so the lane's first block may
    // flip them now (the lane's other blocks may already be in the next group: other scenes).
    __syncthreads();
    if (lb == 0) {
        for (int q = threadIdx.x; q < ns; q += kThreads) {
            const hf_scene& S = scenes[scene_lo + q];
            if (S.flags & HF_FLAG_ACTIVE) write_stats(S, loc[q], HEAT, !ok, s_par[q]);
        }
    }
    __syncthreads();
    return ok;
}

template <bool HEAT, bool TMA>
__global__ void __launch_bounds__(kThreads) k_pcg(const hf_scene* __restrict__ scenes, const TileItem* __restrict__ tiles,
                                                 double dt_d, Workspace ws, const __grid_constant__ GroupTable gt) {
    __shared__ double red[kRedComps * 32];
    __shared__ LocalScene loc[kGroupScenes];
    __shared__ unsigned char s_par[kGroupScenes];
    __shared__ int s_any;
    __shared__ int place[kPlaces];
    __shared__ __align__(8) unsigned long long mbar[2];
    extern __shared__ __align__(128) float sm_raw[];
    float* slots = TMA ? align128_shared(sm_raw) : nullptr;
    unsigned ph = 0u;   // bit s: the phase the next wait on slot s's mbarrier expects (a register, not an array)
    if (TMA && threadIdx.x == 0) {
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int nlb = gridDim.x / gt.lanes;           // blocks per lane (the host launches a multiple of gt.lanes)
    const int lane = blockIdx.x / nlb, lb = blockIdx.x % nlb;
    unsigned* bar = ws.bar + (HEAT ? 0 : kMaxLanes) + lane;
    int* next = ws.lane_next + (HEAT ? 0 : kMaxLanes) + lane;
    unsigned* queue = ws.queue + (HEAT ? 0 : 1);
    unsigned epoch = 0;
    for (;;) {
        if (lb == 0 && threadIdx.x == 0) *(volatile int*)next = (int)atomicAdd(queue, 1u);
        if (!grid_barrier(bar, epoch, ws.err, nlb)) break;
        const int g = *(volatile int*)next;
        if (g >= gt.count) break;
        if (!solve_group<HEAT, TMA>(scenes, tiles, gt.g[g], lb, nlb, bar, epoch, dt_d, ws, red, loc, s_par, &s_any, slots,
                                    mbar, ph, place))
            break;
    }
    // a timed-out barrier leaves the groups that no lane reached unsolved: flag their scenes
    if (blockIdx.x == 0 && *(volatile int*)ws.err) {
        for (int q = 0; q < gt.count; ++q)
            for (int s = gt.g[q].x + (int)threadIdx.x; s < gt.g[q].y; s += kThreads)
                if (scenes[s].flags & HF_FLAG_ACTIVE) scenes[s].state->status |= HF_SCENE_BARRIER_TIMEOUT;
    }
}

const void* pcg_kernel(bool heat, bool tma) {
    return heat ? (const void*)k_pcg<true, false> : tma ? (const void*)k_pcg<false, true> : (const void*)k_pcg<false, false>;
}

size_t pcg_stream_smem(bool tma) { return tma ? 2 * (size_t)kSlotFloats * sizeof(float) + 128 : 0; }

int set_wait_limit(unsigned long long limit_ns, int absent_block) {
    if (cudaMemcpyToSymbol(c_wait_limit_ns, &limit_ns, sizeof limit_ns) != cudaSuccess) return HF_ERR_CUDA;
    if (cudaMemcpyToSymbol(c_absent_block, &absent_block, sizeof absent_block) != cudaSuccess) return HF_ERR_CUDA;
    return brick_set_wait_limit(limit_ns, absent_block);
}

}  // namespace hf
