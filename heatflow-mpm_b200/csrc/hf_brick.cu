// hf_brick.cu -- the CG solves with their state on the chip, one scene per team of blocks.
//
// Same systems, arithmetic and reduction trees as the streaming kernel (hf_cg.cu): the pressure solve -- mean removal,
// Jacobi-preconditioned CG warm-started from p, projection, end of the substep (grid.py:235-251, 94-153) -- and the heat
// solve (heat.py:198-210).  A team of blocks (one per SM) owns a scene's tiles in contiguous runs of whole units; r, A p
// (and D) of a block's cells live in registers, p and x in shared memory, so an iteration moves only what blocks owe each
// other.  A plan of several scenes gives every scene a team of its own and a place in the blocks' common order
// (brick_teams and brick_jobs, hf_api.cu); teams work side by side.
//
// What bounds an iteration: two reductions of the whole scene (p.Ap; r.r and r.z), one halo exchange, and between them the
// issue of some 90 instructions per cell (96^3: 16,300 cycles, of which 7,800 for the exchanges; 45 % issue).  A barrier
// followed by reading the partials costs a release, an atomic, an acquire poll and another round trip (3450 + 2300 cycles
// for 148 blocks of 512 threads).  Here every value carries its own arrival mark instead, so no fence, counter or barrier
// is involved and one trip through L2 does.  Microseconds per pressure iteration, the kernels before -> this one: 32^3
// 6.6 -> 4.6, 75^3 15.8 -> 7.3, 96^3 13.5 -> 8.2, 128^3 33.8 -> 19.8, 160^3 69.2 -> 35.3.
//   * reductions: a block adds its tiles' partials into unit sums and posts each on a 128-byte line of its own as {low
//     word, tag, high word, tag}, self-validating 8-byte halves; every member polls all lines of its team.  A line that
//     is being polled takes one store, of one warp instruction: measured alone, 148 blocks and two values, 1830 to 2400
//     cycles; two stores to the line 2200 to 4300, lines that several blocks write 10,000 and more.
//   * halo: z of the cells on faces that a tile shares with another block's tile, as {z, tag} words that the neighbour
//     polls (again one store for each run of 32).  Each block advances its own copy of p there by the owner's operations
//     on the owner's values.
// Tags name launch (12 bits), job and step (10 bits each), so nothing has to be cleared between launches: every launch
// rewrites each word that its members poll -- a unit's two lines at step 1, the shared faces at the set-up -- so a tag of
// 4096 launches ago is never still there.  A line alternates with the parity of the step: a member posts step s + 2 only
// after step s + 1, which every member posted after reading step s.
#include "hf_cg.cuh"

namespace hf {

constexpr int kFaceBox = 5 * 256 + 4 * 9 * 32 + 4 * 8 * 33;   // floats of one tile's face fractions
constexpr int kBoxY = 5 * 256, kBoxZ = kBoxY + 4 * 9 * 32;
constexpr int kHaloRows = 2 * 8 + 2 * 4 + 2;                  // 32-value rows of a tile's six faces
constexpr int kPollWarps = (kUnits + 31) / 32;                // warps that wait for the other blocks' sums
                                                              // (the others fetch the halo)

// first entry of face f (i-, i+, j-, j+, k-, k+) in a tile's halo slot
__device__ __forceinline__ int face_entry(int f) { return f < 2 ? f * 256 : f < 4 ? 512 + (f - 2) * 128 : 768 + (f - 4) * 32; }

// One tile of the block: nb[f] is the shared-memory offset of the values beyond face f, in the core of another tile of
// the block, in a halo page, or (domain face) the tile's own cells.  Offsets are laid out so that every neighbour of
// cell m lies at nb + m * 256 + (j * 32 | lane), whatever it points to.
struct BrickTile {
    int i0, j0, k0;
    int nb[6];
    int remote;   // bit f: face f borders a tile of another block
    int face;     // offset of the tile's face fractions, or -1: read from the lattices
    int unit;     // all cells in the domain and every fraction between them 1
    int slot;     // first entry of the tile's halo slot
};

__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_halves(ulonglong2* p, double v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | (unsigned)__double2loint(v)),
                 "l"(t | (unsigned)__double2hiint(v))
                 : "memory");
}
__device__ __forceinline__ ulonglong2 ld_halves(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}

// The limit of a wait has passed.  At a job's start others may still be busy with an earlier job: as long as any team of the
// launch has finished an iteration since t0 (its first block notes the time beside err), the wait begins anew from there.
__device__ __forceinline__ unsigned long long extend(int* err, unsigned long long t0, bool start) {
    const unsigned long long beat = ld_relaxed(reinterpret_cast<unsigned long long*>(err + 2));
    if (start && (long long)(beat - t0) > 0) return beat;
    atomicExch(err, 1);
    return 0;
}

// A bounded wait's clock: false once the limit has passed or another block has given up (which sets err).
struct Patience {
    unsigned long long t0 = 0;
    unsigned spins = 0;
    __device__ __forceinline__ bool more(int* err, bool start) {
        if (++spins & 63u) return true;
        if (*(volatile int*)err) return false;
        const unsigned long long now = global_timer_ns();
        if (!t0) t0 = now;
        if ((long long)(now - t0) <= (long long)c_wait_limit_ns) return true;
        t0 = extend(err, t0, start);
        return t0 != 0;
    }
};

// The warp sums of K values per lane, value by value the butterfly of offsets 16, 8, 4, 2, 1: while more than one value is
// left, the lanes of a pair share them (each keeps half and adds the other's), which adds the same numbers in the same
// order as K separate butterflies, with half the exchanges or fewer.  Returns the value's index; its sum is in v[0].
template <int K, int P, int OFF>
__device__ __forceinline__ void fold(double* v, int lane, int& index) {
    if constexpr (OFF > 0) {
        if constexpr (P == 1) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], OFF);
            fold<1, 1, OFF / 2>(v, lane, index);
        } else {
            constexpr int H = P / 2;
            const bool hi = lane & OFF;
#pragma unroll
            for (int i = 0; i < H; ++i) {
                if (i >= K) continue;
                const double a = v[i], b = i + H < K ? v[i + H] : 0.0;
                v[i] = (hi ? b : a) + __shfl_xor_sync(0xffffffffu, hi ? a : b, OFF);
            }
            index += hi ? H : 0;
            fold<(K < H ? K : H), H, OFF / 2>(v, lane, index);
        }
    }
}
__host__ __device__ constexpr int pow2_above(int k) { return k <= 1 ? 1 : 2 * pow2_above((k + 1) / 2); }

// a / b: Newton's iteration for 1 / b from its binary32 value, then the quotient with Markstein's correction (IBM J. Res.
// Dev. 34(1), 1990; the remainder a - q b is exact with one FMA).  150 cycles from operands to result instead of 410 to 700
// for the operator, and the scalars of an iteration wait for two of them.  Markstein's result, that the corrected quotient is
// rounded correctly, needs a correctly rounded 1 / b, which the iteration does not reach when every bit of b's significand is
// set (2^k over such a b came out one place low); two steps do not prove it for every other b, so hf_k_quotient compares
// with the operator.  Those b, and operands outside [2^-100, 2^100], take the operator.
__device__ __forceinline__ double quotient(double a, double b) {
    const double ab = fabs(b), aa = fabs(a);
    const bool ones = __double2loint(b) == -1 && (__double2hiint(b) & 0xfffff) == 0xfffff;
    if (!(ab >= 0x1p-100 && ab <= 0x1p100 && aa >= 0x1p-100 && aa <= 0x1p100) || ones) return a / b;
    double y = (double)__frcp_rn((float)b);
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    const double q = a * y;
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// div_rn of four values at once: one test of their range instead of four.  Zeros (every cell outside the domain has one)
// stay on the short way: their quotient comes out as zero there too.
__device__ __forceinline__ void div_rn4(float (&x)[4], const DivBy& d) {
    float low[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) low[m] = x[m] == 0.0f ? 1.0f : fabsf(x[m]);
    const float lo = fminf(fminf(low[0], low[1]), fminf(low[2], low[3]));
    const float hi = fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3])));
    if (lo >= 0x1p-96f && hi <= 0x1p96f) {   // a NaN among them passes through both ways
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float q = __fmaf_rn(x[m], d.zh, __fmul_rn(x[m], d.zl));
            x[m] = __fmaf_rn(__fmaf_rn(-q, d.y, x[m]), d.zh, q);
        }
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = div_rn(x[m], d);
    }
}

// a job's word in ws.arrive: members that are done with it; a member gave up, and the scene's parity that it started from
constexpr unsigned kArrived = 0xffffu, kGaveUp = 1u << 30, kParity = 1u << 31;

// The scenes of a launch of which any member gave up are timeouts, whatever their first blocks found: not counted, old parity.
// (A function of its own: in line, its registers made an iteration at 96^3 5 % slower.)
__device__ __noinline__ void take_back(const hf_scene* scenes, const unsigned* arrive, const int4* of, int jobs, int only, bool heat) {
    __threadfence();
    for (int q = 0; q < jobs; ++q) {
        const unsigned a = *(volatile const unsigned*)(arrive + q);
        if (!(a & kGaveUp)) continue;
        volatile hf_scene_state* st = scenes[jobs == 1 ? only : of[q].x].state;
        st->status |= HF_SCENE_BARRIER_TIMEOUT;
        if (!heat && st->parity != (int)(a / kParity)) {
            st->parity ^= 1;
            st->substeps -= 1;
        }
    }
}

// A block's place in a team.  A block owns at most as many units as tiles.
constexpr int kLines = kBrickWideTiles;        // lines of a block and parity
struct Team {
    int units, mine;                           // units of the scene and of this block,
    const int* begin;                          // the first tile of each of these (and the end)
    ulonglong2* post;                          // this block's lines (two parities)
    const ulonglong2* poll;                    // the line of unit threadIdx.x
    unsigned base;                             // launch and job part of the tags
    int* err;
};

// The scene sums of K components from the tile partials in red[(c * 8 + warp) * NT + tile], handed to `derive` in the first
// thread, which leaves what the block needs in shared memory (every thread deriving it for itself made 96^3 5 % slower).
// `before` is what the warps that do not wait for the sums do meanwhile.  False, in every thread, when a wait of any
// thread gave up (bad).
template <int K, int NT, class Before, class Derive>
__device__ __forceinline__ bool exchange(const Team& team, int nt, unsigned& step, const double* red, double* tsum,
                                         double (*sums)[8], int& bad, Before before, Derive derive) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    ++step;
    const unsigned tag = team.base | (step & 0x3ffu);
    __syncthreads();
    if (warp == 0 && !(step == 1 && (int)blockIdx.x == c_absent_block)) {
        // tile partials (8 warps in order), then the unit sums (tiles in order): lane 4 u + c has component c of unit u,
        // so a unit's line is written by one instruction
        // (absent tiles as +0.0, which changes nothing).  All loads come before the additions.
        for (int tile = lane; tile < nt; tile += 32) {
            double w[K][8];
#pragma unroll
            for (int c = 0; c < K; ++c)
#pragma unroll
                for (int q = 0; q < 8; ++q) w[c][q] = red[(c * 8 + q) * NT + tile];
#pragma unroll
            for (int c = 0; c < K; ++c) {
                double s = 0.0;
#pragma unroll
                for (int q = 0; q < 8; ++q) s += w[c][q];
                tsum[c * NT + tile] = s;
            }
        }
        __syncwarp();
        for (int u = lane >> 2; u < team.mine; u += 8) {
            const int c = lane & 3, a = team.begin[u], e = team.begin[u + 1];
            if (c >= K) continue;
            constexpr int kAtOnce = NT <= 15 ? NT : 12;
            double s = 0.0;
            for (int q0 = a; q0 < e; q0 += kAtOnce) {
                double v[kAtOnce];
#pragma unroll
                for (int q = 0; q < kAtOnce; ++q) v[q] = q0 + q < e ? tsum[c * NT + q0 + q] : 0.0;
#pragma unroll
                for (int q = 0; q < kAtOnce; ++q) s += v[q];
            }
            st_halves(team.post + ((step & 1u) * kLines + u) * 8 + c, s, tag);
            // The line of the even steps as well, under a tag that nobody looks for there: a solve may end before its first
            // even step, and what an older launch left would come up again when the launch number has gone round.
            if (step == 1) st_halves(team.post + u * 8 + c, s, tag);
        }
    }
    if (warp >= kPollWarps) {
        before();
    } else {
        double v[K];
#pragma unroll
        for (int c = 0; c < K; ++c) v[c] = 0.0;
        // The warp leaves the loop together, by vote: lanes that left it one by one would stay apart until the next barrier
        // and issue every following shuffle group by group (250 cycles each instead of 33).
        const ulonglong2* line = team.poll + (step & 1u) * kLines * 8;
        bool here = t >= team.units;
        Patience patience;
        for (;;) {
            if (!here) {
                ulonglong2 q[K];
#pragma unroll
                for (int c = 0; c < K; ++c) q[c] = ld_halves(line + c);
                here = true;
#pragma unroll
                for (int c = 0; c < K; ++c) {
                    here = here && (unsigned)(q[c].x >> 32) == tag && (unsigned)(q[c].y >> 32) == tag;
                    v[c] = __hiloint2double((int)(unsigned)q[c].y, (int)(unsigned)q[c].x);
                }
            }
            if (__all_sync(0xffffffffu, here)) break;
            if (__any_sync(0xffffffffu, !patience.more(team.err, step == 1))) {
                bad = 1;
                break;
            }
        }
#pragma unroll
        for (int c = 0; c < K; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
            if (lane == 0) sums[c][warp] = v[c];
        }
        asm volatile("bar.sync 15, %0;" ::"n"(kPollWarps * 32) : "memory");
        if (t == 0) {
            double tot[K];
#pragma unroll
            for (int c = 0; c < K; ++c) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < kPollWarps; ++w) s += sums[c][w];
                tot[c] = s;
            }
            derive(tot);
        }
    }
    return !__syncthreads_or(bad);
}

// G groups of 256 threads with up to Q tiles each.  With one tile a thread keeps all of its cells' state in registers (p also
// in shared memory, for the neighbours); up to three it keeps D; beyond, D of a unit tile follows from the number of a
// cell's faces, and other tiles read it back.
// Q = 0, for large scenes: only p stays on the chip.  r, A p and x are read and written where they are used, by the thread
// that owns the cell (28 bytes of L2 traffic per cell and iteration; the streaming kernel moves 60 and p's halo from HBM).
template <int G, int Q, bool HEAT>
__global__ void __launch_bounds__(256 * G, 1)
    k_brick(const hf_scene* __restrict__ scenes, const TileItem* __restrict__ tiles, double dt_d, Workspace ws, BrickLaunch bl) {
    constexpr bool kWide = Q == 0;
    constexpr int QR = kWide ? 1 : Q;                         // tiles a thread holds at a time
    constexpr int NT = kWide ? kBrickWideTiles : G * Q;
    constexpr int kWarps = 8 * G, kRowWarps = kWarps - kPollWarps;
    constexpr int kRowsEach = kWide ? 16 : G == 4 ? 3 : Q <= 2 ? 6 : 10;   // halo rows that a warp keeps while the sums are on their way
    constexpr bool kKeepD = !kWide && Q <= 3, kKeepX = NT <= 2;
    constexpr bool kLattice = kWide || NT > 9;                // general tiles may find no box for their fractions
    extern __shared__ __align__(16) float sm[];   // p, x (1024 floats a tile each), halo pages, face boxes
    __shared__ BrickTile tt[NT];
    __shared__ int2 rows[NT * kHaloRows];         // (entry in the neighbour's slot, shared offset; bit 30: a k face)
    __shared__ double red[3 * NT * 8];
    __shared__ double tsum[3 * NT];
    __shared__ int ubegin[kLines + 1];
    __shared__ float kface[2 * 32];               // values of the run's two k faces on their way out
    __shared__ double sums[3][8];
    __shared__ LocalScene Ls;
    __shared__ hf_scene Ss;
    __shared__ float dtab[8];
    __shared__ int s_count[6];                    // i planes, j slots, k columns, rows, face boxes in use; [5]: s_gave_up
    int& s_gave_up = s_count[5];                  // a job of this block did not end for a wait that gave up (thread 0)
    const int g = threadIdx.x >> 8, lt = threadIdx.x & 255, lane = lt & 31, row = lt >> 5, warp = threadIdx.x >> 5;
    int* const err = reinterpret_cast<int*>(ws.brick + 2);
    const unsigned launch = *(volatile unsigned*)ws.brick;
    const int X = kWide ? 0 : bl.tiles * 1024;    // x follows p (wide: takes p's place at the end)
    const int pages = bl.tiles * (kWide ? 1024 : 2048), boxes = pages + bl.pages * 1024;
    int bad = 0;                                  // a wait of this thread gave up
    int left = -1, left_nb = 0;                   // the job before and its blocks
    if (threadIdx.x == 0) s_gave_up = 0;

    for (int job = 0; job < bl.jobs; ++job) {
        const int4 J = bl.jobs == 1 ? bl.job0 : ws.jobs[job];   // scene, first block, blocks
        if ((int)blockIdx.x < J.y || (int)blockIdx.x >= J.y + J.z) continue;
        // the scene's record in shared memory: its pointers are fetched again and again, and a trip to L2 before every access
        // made the set-up and the projection several times slower
        for (int w = threadIdx.x; w < (int)(sizeof(hf_scene) / sizeof(int)); w += 256 * G)
            reinterpret_cast<int*>(&Ss)[w] = reinterpret_cast<const int*>(scenes + J.x)[w];
        const hf_scene& S = Ss;
        const bool leader = (int)blockIdx.x == J.y;
        if (__syncthreads_or(*(volatile int*)err)) {   // a wait gave up earlier in this launch: the scene stays unsolved
            if (leader && threadIdx.x == 0) S.state->status = (HEAT ? 0 : S.state->status) | HF_SCENE_BARRIER_TIMEOUT;
            continue;
        }
        Team team;
        const int b = (int)blockIdx.x - J.y, tb = ws.tile_begin[J.x];
        const int T = ws.tile_begin[J.x + 1] - tb;
        team.units = unit_count(T);
        const int u0 = unit_first(team.units, J.z, b), u1 = unit_first(team.units, J.z, b + 1);
        const int c0 = unit_first(T, team.units, u0), c1 = unit_first(T, team.units, u1), nt = c1 - c0;
        team.mine = u1 - u0;
        team.begin = ubegin;
        team.post = ws.mail + (size_t)blockIdx.x * 2 * kLines * 8;
        {
            // the owner of unit t and the unit's place among its units
            const int t = (int)threadIdx.x < team.units ? threadIdx.x : 0, o = ((t + 1) * J.z - 1) / team.units;
            team.poll = ws.mail + ((size_t)(J.y + o) * 2 * kLines + t - unit_first(team.units, J.z, o)) * 8;
        }
        team.base = launch << 20 | (unsigned)job << 10;
        team.err = err;
        unsigned step = 0, pub = 0;
        bool ok = true;
        const int n = S.n, par = S.state->parity;
        const float h = (float)S.h, hh = __fmul_rn(h, h);
        const DivBy hhd = div_by(hh);
        const float c_dt = __fdiv_rn((float)dt_d, hh);
        float* const xg = HEAT ? S.T[par ^ 1] : S.p;
        float* const Dg = HEAT ? S.hdiag : S.pdiag;
        const int ti = (n + kTI - 1) / kTI, tj = (n + kTJ - 1) / kTJ, tk = (n + kTK - 1) / kTK;

        // ------------------------------------------------------------------------------------ the block's tiles
        if (threadIdx.x < 5) s_count[threadIdx.x] = 0;
        if ((int)threadIdx.x <= team.mine) ubegin[threadIdx.x] = unit_first(T, team.units, u0 + threadIdx.x) - c0;
        if (threadIdx.x < 7) dtab[threadIdx.x] = __fdiv_rn(hh, maxf_((float)threadIdx.x, 1.0e-12f));
        __syncthreads();
        if (threadIdx.x < nt) {
            const int q = threadIdx.x, c = c0 + q;
            const TileItem it = tiles[tb + c];
            BrickTile t;
            t.i0 = it.i0;
            t.j0 = it.j0;
            t.k0 = it.k0;
            t.slot = (tb + c) * kHaloEntries;
            t.remote = 0;
            t.face = -1;
            t.unit = !HEAT && it.i0 + kTI <= n && it.j0 + kTJ <= n && it.k0 + kTK <= n;
            const bool there[6] = {it.i0 > 0, it.i0 / kTI + 1 < ti, it.j0 > 0, it.j0 / kTJ + 1 < tj, it.k0 > 0, it.k0 / kTK + 1 < tk};
            const int away[6] = {-tk, tk, -tk * ti, tk * ti, -1, 1};
            // offsets within the neighbour's core, and within the tile's own (domain faces: the cell itself)
            const int far[6] = {768, 0, 224, 0, 31, 0}, own[6] = {0, 768, 0, 224, 0, 31};
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                const int o = c + away[f];
                if (!there[f]) {
                    t.nb[f] = q * 1024 + own[f];
                } else if (o >= c0 && o < c1) {
                    t.nb[f] = (o - c0) * 1024 + far[f];
                } else {
                    t.remote |= 1 << f;
                    const int kind = f >> 1, at = atomicAdd(&s_count[kind], 1);
                    // a page holds 4 planes (i faces), 8 slots of a row per m (j faces) or 32 columns (k faces)
                    const int room = kind == 0 ? 4 * bl.i_pages : kind == 1 ? 8 * bl.j_pages : 32 * (bl.pages - bl.i_pages - bl.j_pages);
                    if (at >= room) {
                        atomicExch(err, 1);   // cannot happen: the launch sizes the pages for its longest run
                        t.nb[f] = q * 1024 + own[f];
                        continue;
                    }
                    const int page = pages + (kind == 0 ? at / 4 : kind == 1 ? bl.i_pages + at / 8 : bl.i_pages + bl.j_pages + at / 32) * 1024;
                    t.nb[f] = page + (kind == 0 ? (at % 4) * 256 : kind == 1 ? (at % 8) * 32 : at % 32);
                    const int src = (tb + o) * kHaloEntries + face_entry(f ^ 1), count = kind == 0 ? 8 : kind == 1 ? 4 : 1;
                    const int r0 = atomicAdd(&s_count[3], count);
                    for (int r = 0; r < count; ++r)
                        rows[r0 + r] = make_int2(src + r * 32, kind == 0 ? t.nb[f] + r * 32 : kind == 1 ? t.nb[f] + r * 256
                                                                                                         : t.nb[f] | 1 << 30);
                }
            }
            tt[q] = t;
        }
        if (left >= 0 && threadIdx.x == 0) {
            // everyone has read this block's last sums of the job before: its lines may be written again
            Patience patience;
            while ((ld_acquire_u32(ws.arrive + left) & kArrived) < (unsigned)left_nb)
                if (!patience.more(err, true)) {
                    bad = 1;
                    break;
                }
        }
        // the pressure rhs mean (grid.py:238-241) from the divergence stage's chunk sums: 256 threads in strides, warp
        // butterfly, 8 warps in order
        float mean = 0.0f;
        __syncthreads();
        if (!HEAT) {
            double m = 0.0;
            if (threadIdx.x < kThreads)
                for (int c = ws.chunk_begin[J.x] + threadIdx.x; c < ws.chunk_begin[J.x + 1]; c += kThreads) m += ws.mean_part[c];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
            __syncthreads();
            if (lane == 0 && warp < 8) sums[0][warp] = m;
            __syncthreads();
            m = 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q) m += sums[0][q];
            mean = __double2float_rn(m / ((double)n * n * n));
        }
        const int nrows = s_count[3];
        auto post = [&](const BrickTile& T, const float (&v)[4], unsigned tag) {
            const int rem = T.remote;
            if (!rem) return;
            unsigned long long* to = ws.halo + T.slot;
            const unsigned long long mark = (unsigned long long)tag << 32;
            auto put = [&](int e, float x) { st_relaxed(to + e, mark | __float_as_uint(x)); };
            if (rem & 1) put(lt, v[0]);
            if (rem & 2) put(256 + lt, v[3]);
            if ((rem & 4) && row == 0)
#pragma unroll
                for (int m = 0; m < 4; ++m) put(512 + m * 32 + lane, v[m]);
            if ((rem & 8) && row == 7)
#pragma unroll
                for (int m = 0; m < 4; ++m) put(640 + m * 32 + lane, v[m]);
            // a k face (the run's first or last) comes from eight warps: gathered here, sent by one (post_k, after a barrier)
            if ((rem & 16) && lane == 0)
#pragma unroll
                for (int m = 0; m < 4; ++m) kface[m * 8 + row] = v[m];
            if ((rem & 32) && lane == 31)
#pragma unroll
                for (int m = 0; m < 4; ++m) kface[32 + m * 8 + row] = v[m];
        };
        auto post_k = [&](unsigned tag) {
            const int e = warp - kPollWarps;
            if (e > 1) return;
            const BrickTile& T = tt[e ? nt - 1 : 0];
            if (T.remote & (16 << e))
                st_relaxed(ws.halo + T.slot + 768 + e * 32 + lane, (unsigned long long)tag << 32 | __float_as_uint(kface[e * 32 + lane]));
        };
        // The halo's rows.  fetch: the warps that do not wait for the sums wait for theirs, up to kRowsEach rows each, into
        // registers.  take: every value goes to its place through apply(place, value).
        float ahead[kRowsEach];
        auto await = [&](int r, unsigned tag, unsigned long long v) {
            const unsigned long long* from = ws.halo + rows[r].x + lane;
            // A neighbour whose last sums told it that the solve has ended may already have put x in z's place.  That is as
            // good as z here: this block is about to learn the same, and z is not used any more.
            const unsigned after = team.base | ((tag + 1) & 0x3ffu);
            Patience patience;
            while (__any_sync(0xffffffffu, (unsigned)(v >> 32) != tag && (unsigned)(v >> 32) != after)) {   // together
                if (__any_sync(0xffffffffu, !patience.more(err, (tag & 0x3ffu) == 1))) {
                    bad = 1;
                    break;
                }
                v = ld_relaxed(from);
            }
            return __uint_as_float((unsigned)v);
        };
        auto fetch = [&](unsigned tag) {
            post_k(tag);
            unsigned long long v[kRowsEach];
#pragma unroll
            for (int u = 0; u < kRowsEach; ++u) {
                const int r = warp - kPollWarps + u * kRowWarps;
                v[u] = r < nrows ? ld_relaxed(ws.halo + rows[r].x + lane) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < kRowsEach; ++u) {
                const int r = warp - kPollWarps + u * kRowWarps;
                if (r < nrows) ahead[u] = await(r, tag, v[u]);
            }
            if (bl.jobs > 1 && leader && threadIdx.x == 32 * kPollWarps)   // for who waits for this team's blocks (extend)
                st_relaxed(reinterpret_cast<unsigned long long*>(ws.brick + 4), global_timer_ns());
        };
        auto take = [&](unsigned tag, auto apply) {
            auto place = [&](int r) {
                const int at = rows[r].y;
                return (at >> 30) & 1 ? (at & 0x3fffffff) + (lane >> 3) * 256 + (lane & 7) * 32 : at + lane;
            };
            if (warp >= kPollWarps) {
#pragma unroll
                for (int u = 0; u < kRowsEach; ++u) {
                    const int r = warp - kPollWarps + u * kRowWarps;
                    if (r < nrows) apply(sm[place(r)], ahead[u]);
                }
            }
            for (int r = kRowWarps * kRowsEach + warp; r < nrows; r += kWarps)
                apply(sm[place(r)], await(r, tag, ld_relaxed(ws.halo + rows[r].x + lane)));
        };

        // the first of a tile's four cells, and which of them the domain has
        auto first_cell = [&](const BrickTile& T, int& cells) {
            const int j = T.j0 + row, k = T.k0 + lane;
            cells = j < n && k < n ? min(4, n - T.i0) : 0;
            return (T.i0 * n + j) * n + k;
        };
        // Face coefficients around two cells (i, j, k) and (i + 1, j, k) from the lattices: x faces i .. i + 2, low and high
        // y and z faces; 0 where a face has no cell on one side, so that its term drops out.  Two cells at a time: their
        // loads are in flight together and fit the registers.  (Taking the z neighbours from the next lane saved a third
        // of the loads and made the set-up a quarter slower: the shuffles wait for the loads one by one.)
        const int nn = n * n;
        const float* const cx = HEAT ? S.hkx : S.ax;
        const float* const cy = HEAT ? S.hky : S.ay;
        const float* const cz = HEAT ? S.hkz : S.az;
        auto coefficients = [&](int i, int j, int k, float (&fx)[3], float (&fy)[4], float (&fz)[4]) {
            const bool in = j < n && k < n;
#pragma unroll
            for (int a = 0; a < 3; ++a) fx[a] = in && i + a > 0 && i + a < n ? cx[uidx_(n, i + a, j, k)] : 0.0f;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const bool im = in && i + a < n;
                fy[a] = im && j > 0 ? cy[vidx_(n, i + a, j, k)] : 0.0f;
                fy[2 + a] = im && j < n - 1 ? cy[vidx_(n, i + a, j + 1, k)] : 0.0f;
                fz[a] = im && k > 0 ? cz[widx_(n, i + a, j, k)] : 0.0f;
                fz[2 + a] = im && k < n - 1 ? cz[widx_(n, i + a, j, k + 1)] : 0.0f;
            }
        };
        // the cell values (or flags) of the same two cells and their neighbours: i - 1 .. i + 2, low and high j and k; 0
        // outside the domain
        auto around = [&](const auto* from, int i, int j, int k, auto (&vi)[4], auto (&vj)[4], auto (&vk)[4]) {
            const bool in = j < n && k < n;
            const int t = (i * n + j) * n + k;
#pragma unroll
            for (int a = 0; a < 4; ++a) vi[a] = in && i + a > 0 && i + a <= n ? from[t + (a - 1) * nn] : 0;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const bool im = in && i + a < n;
                vj[a] = im && j > 0 ? from[t + a * nn - n] : 0;
                vj[2 + a] = im && j < n - 1 ? from[t + a * nn + n] : 0;
                vk[a] = im && k > 0 ? from[t + a * nn - 1] : 0;
                vk[2 + a] = im && k < n - 1 ? from[t + a * nn + 1] : 0;
            }
        };
        // one face's term of the stencil; heat: a fixed neighbour enters as kappa_f x_c (heat.py:55-91)
        auto term = [](float c, bool fixed, float xc, float xn) { return __fmul_rn(c, HEAT && fixed ? xc : __fsub_rn(xc, xn)); };
        // the warp's sums of K components of its tiles (one: q, wide; else the group's) go to red
        auto stash = [&](int q, auto& part) {
            constexpr int N = (int)(sizeof(part) / sizeof(double)), P = pow2_above(N);
            static_assert(P <= 32, "one value per lane at most");
            int index = 0;
            fold<N, P, 16>(part, lane, index);
            const int at = kWide ? q : G * (index % QR) + g;
            if (index < N && (lane & (32 / P - 1)) == 0 && at < nt) red[(index / QR * 8 + row) * NT + at] = part[0];
        };
        // ------------------------------------------------------------------------------------ set-up
        float r[4 * QR], ap[4 * QR], dg[kKeepD ? 4 * QR : 1], xr[kKeepX ? 4 * QR : 1], pr[kKeepX ? 4 * QR : 1];
        const int turns = kWide ? (nt - g + G - 1) / G : Q;   // of the loops over a group's tiles; unrolled unless wide
        // heat: byte m: which of cell m's neighbours (in the faces' order) and, bit 6, the cell itself are fixed
        unsigned fixed[HEAT ? QR : 1];
        {
            // x0, b, D, r0 = b - A x0, z0 = D r0; pressure: x0 = p, b = rhs - mean, and a tile with a fraction other than 1
            // is general; heat: x0 = the advected T, b = hrhs
            double part[3 * QR];
#pragma unroll QR
            for (int turn = 0; turn < turns; ++turn) {
                const int s = kWide ? 0 : turn, q = G * turn + g;
                part[s] = part[QR + s] = part[2 * QR + s] = 0.0;
                float z4[4];
                if (q < nt) {
                    const int j = tt[q].j0 + row, k = tt[q].k0 + lane;
                    bool one = true;
#pragma unroll
                    for (int m0 = 0; m0 < 4; m0 += 2) {
                        const int i0 = tt[q].i0 + m0, t0 = (i0 * n + j) * n + k;
                        float fx[3], fy[4], fz[4], xi[4], xj[4], xk[4], bv[2];
                        int gi[4] = {}, gj[4] = {}, gk[4] = {};
                        coefficients(i0, j, k, fx, fy, fz);
                        around(xg, i0, j, k, xi, xj, xk);
                        if (HEAT) around(S.cell_flags, i0, j, k, gi, gj, gk);
                        const bool ok2[2] = {j < n && k < n && i0 < n, j < n && k < n && i0 + 1 < n};
#pragma unroll
                        for (int a = 0; a < 2; ++a) bv[a] = ok2[a] ? (HEAT ? S.hrhs : S.rhs)[t0 + a * nn] : 0.0f;
#pragma unroll
                        for (int a = 0; a < 2; ++a) {
                            const int m = m0 + a, e = s * 4 + m, i = i0 + a;
                            const float xc = xi[a + 1];
                            const float af[6] = {fx[a], fx[a + 1], fy[a], fy[2 + a], fz[a], fz[2 + a]};
                            float sa = af[0];
#pragma unroll
                            for (int f = 1; f < 6; ++f) sa = __fadd_rn(sa, af[f]);
                            const int mask = (gi[a] & 1) | (gi[a + 2] & 1) << 1 | (gj[a] & 1) << 2 | (gj[2 + a] & 1) << 3 |
                                             (gk[a] & 1) << 4 | (gk[2 + a] & 1) << 5 | (gi[a + 1] & 1) << 6;
                            if (HEAT) fixed[s] = m ? fixed[s] | (unsigned)mask << (8 * m) : (unsigned)mask;
                            float acc = term(af[0], mask & 1, xc, xi[a]);
                            acc = __fadd_rn(acc, term(af[1], mask & 2, xc, xi[a + 2]));
                            acc = __fadd_rn(acc, term(af[2], mask & 4, xc, xj[a]));
                            acc = __fadd_rn(acc, term(af[3], mask & 8, xc, xj[2 + a]));
                            acc = __fadd_rn(acc, term(af[4], mask & 16, xc, xk[a]));
                            acc = __fadd_rn(acc, term(af[5], mask & 32, xc, xk[2 + a]));
                            float d = 0.0f, rv = 0.0f, z = 0.0f;
                            if (ok2[a]) {
                                if (mean != 0.0f) {
                                    bv[a] = __fsub_rn(bv[a], mean);
                                    S.rhs[t0 + a * nn] = bv[a];
                                }
                                if (HEAT) {   // k_heat_diag; identity rows on fixed cells
                                    d = mask & 64 ? 1.0f : __fdiv_rn(1.0f, __fadd_rn(1.0f, __fmul_rn(c_dt, sa)));
                                    rv = __fsub_rn(bv[a], mask & 64 ? xc : __fadd_rn(xc, __fmul_rn(c_dt, acc)));
                                } else {      // k_jacobi
                                    d = __fdiv_rn(hh, maxf_(sa, 1.0e-12f));
                                    rv = __fsub_rn(bv[a], div_rn(acc, hhd));
                                    one = one && (af[0] == 1.0f || i == 0) && (af[1] == 1.0f || i == n - 1) && (af[2] == 1.0f || j == 0) &&
                                          (af[3] == 1.0f || j == n - 1) && (af[4] == 1.0f || k == 0) && (af[5] == 1.0f || k == n - 1);
                                }
                                z = __fmul_rn(d, rv);
                                if (kWide) S.cg_r[t0 + a * nn] = rv;
                                if (!kKeepD) Dg[t0 + a * nn] = d;
                                part[s] += (double)bv[a] * (double)bv[a];
                                part[QR + s] += (double)rv * (double)rv;
                                part[2 * QR + s] += (double)rv * (double)z;
                            }
                            r[e] = rv;
                            ap[e] = 0.0f;
                            if (kKeepD) dg[e] = d;
                            z4[m] = z;
                            if (kKeepX) {
                                xr[e] = xc;
                                pr[e] = z;
                            } else if (!kWide) {
                                sm[X + q * 1024 + m * 256 + lt] = xc;
                            }
                            sm[q * 1024 + m * 256 + lt] = z;
                        }
                        asm volatile("" ::: "memory");   // the next two cells' loads stay behind
                    }
                    if (!one) tt[q].unit = 0;
                    if (HEAT && kWide) {
                        int cells;
                        const int t = first_cell(tt[q], cells);
                        if (cells > 0) S.cg_z[t] = __uint_as_float(fixed[0]);
                    }
                    post(tt[q], z4, team.base | (pub + 1));
                } else {
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        r[s * 4 + m] = ap[s * 4 + m] = 0.0f;
                        if (kKeepD) dg[s * 4 + m] = 0.0f;
                        if (kKeepX) xr[s * 4 + m] = pr[s * 4 + m] = 0.0f;
                    }
                }
                if (kWide) stash(q, part);
            }
            ++pub;
            if (!kWide) stash(g, part);
        }
        {
            ok = exchange<3, NT>(team, nt, step, red, tsum, sums, bad, [&] { fetch(team.base | pub); },
                                 [&](const double (&tot)[3]) {
                                     init_scalars(Ls, S, HEAT, tot, n * n * n);
                                     Ls.mean = (double)mean;
                                 });
        }
        // face fractions of the general tiles, zero where a face has no cell on one side (those terms drop out)
        for (int q = g; !HEAT && q < nt; q += G) {
            if (tt[q].unit) continue;   // uniform in the group
            if (lt == 0) {
                const int at = atomicAdd(&s_count[4], 1);
                tt[q].face = at < bl.boxes ? boxes + at * kFaceBox : -1;
            }
            asm volatile("bar.sync %0, 256;" ::"r"(g + 1) : "memory");
            const int to = tt[q].face, i0 = tt[q].i0, j0 = tt[q].j0, k0 = tt[q].k0;
            if (to < 0) continue;
            for (int e = lt; e < kFaceBox; e += 256) {
                float v = 0.0f;
                if (e < kBoxY) {
                    const int i = i0 + (e >> 8), j = j0 + ((e >> 5) & 7), k = k0 + (e & 31);
                    if (i > 0 && i < n && j < n && k < n) v = __ldg(S.ax + uidx_(n, i, j, k));
                } else if (e < kBoxZ) {
                    const int w = e - kBoxY, i = i0 + w / 288, j = j0 + (w % 288) / 32, k = k0 + (w & 31);
                    if (j > 0 && i < n && j < n && k < n) v = __ldg(S.ay + vidx_(n, i, j, k));
                } else {
                    const int w = e - kBoxZ, i = i0 + w / 264, j = j0 + (w % 264) / 33, k = k0 + w % 33;
                    if (k > 0 && i < n && j < n && k < n) v = __ldg(S.az + widx_(n, i, j, k));
                }
                sm[to + e] = v;
            }
        }
        __syncthreads();
        bool live = ok && Ls.live;
        int kit = 0;
        float beta = 0.0f;

        // D of the four cells of a tile when it is not kept (a unit tile's from the number of faces in the domain)
        auto diag = [&](const BrickTile& T, int s, float (&d)[4]) {
            if constexpr (kKeepD) {
#pragma unroll
                for (int m = 0; m < 4; ++m) d[m] = dg[s * 4 + m];
            } else {
                const int j = T.j0 + row, k = T.k0 + lane;
                if (T.unit) {
                    const int c = 6 - (j == 0) - (j == n - 1) - (k == 0) - (k == n - 1);
                    d[1] = d[2] = dtab[c];
                    d[0] = dtab[c - (T.i0 == 0)];
                    d[3] = dtab[c - (T.i0 + 4 == n)];
                } else {
                    const bool in = j < n && k < n;
                    const float* from = Dg + (T.i0 * n + j) * n + k;
#pragma unroll
                    for (int m = 0; m < 4; ++m) d[m] = in && T.i0 + m < n ? from[m * nn] : 0.0f;
                }
            }
        };

        // ------------------------------------------------------------------------------------ iterations
        while (live) {
            ++kit;
            // p = z + beta p: the halo's copies and the block's own cells (the first p is z, placed by the set-up)
            take(team.base | (pub & 0x3ffu), [&](float& pb, float z) { pb = kit == 1 ? z : __fadd_rn(z, __fmul_rn(beta, pb)); });
            if (kit > 1) {
#pragma unroll QR
                for (int turn = 0; turn < turns; ++turn) {
                    const int s = kWide ? 0 : turn, q = G * turn + g;
                    if (q >= nt) continue;
                    float d[4], rv[4];
                    diag(tt[q], s, d);
                    float* core = sm + q * 1024 + lt;
                    int cells = 0;
                    const int t = kWide ? first_cell(tt[q], cells) : 0;
#pragma unroll
                    for (int m = 0; m < 4; ++m) rv[m] = !kWide ? r[s * 4 + m] : m < cells ? S.cg_r[t + m * nn] : 0.0f;
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const float pv = __fadd_rn(__fmul_rn(d[m], rv[m]), __fmul_rn(beta, kKeepX ? pr[s * 4 + m] : core[m * 256]));
                        core[m * 256] = pv;
                        if (kKeepX) pr[s * 4 + m] = pv;
                    }
                }
            }
            __syncthreads();
            double pAp[QR];
#pragma unroll QR
            for (int turn = 0; turn < turns; ++turn) {
                const int s = kWide ? 0 : turn, q = G * turn + g;
                pAp[s] = 0.0;
                if (q >= nt) continue;
                const BrickTile& T = tt[q];
                const int core = q * 1024 + lt;
                const float* lo_j = sm + (row == 0 ? T.nb[2] + lane : core - 32);
                const float* hi_j = sm + (row == 7 ? T.nb[3] + lane : core + 32);
                const float* lo_k = sm + (lane == 0 ? T.nb[4] + row * 32 : core - 1);
                const float* hi_k = sm + (lane == 31 ? T.nb[5] + row * 32 : core + 1);
                float p[6];   // the column i0 - 1 .. i0 + 4
                p[0] = sm[T.nb[0] + lt];
                p[5] = sm[T.nb[1] + lt];
#pragma unroll
                for (int m = 0; m < 4; ++m) p[m + 1] = kKeepX ? pr[s * 4 + m] : sm[core + m * 256];
                float a[4];
                if constexpr (HEAT) {
                    // heat.py:94-105: identity rows on fixed cells.  The solve takes an iteration or two, so the diffusivities
                    // come from the lattices
                    const int j = T.j0 + row, k = T.k0 + lane;
                    if (kWide) {
                        int cells;
                        const int t = first_cell(T, cells);
                        fixed[0] = cells > 0 ? __float_as_uint(S.cg_z[t]) : 0u;
                    }
#pragma unroll
                    for (int m0 = 0; m0 < 4; m0 += 2) {
                        float fx[3], fy[4], fz[4];
                        coefficients(T.i0 + m0, j, k, fx, fy, fz);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int m = m0 + e;
                            const unsigned mask = fixed[s] >> (8 * m);
                            const float pc = p[m + 1];
                            float acc = term(fx[e], mask & 1, pc, p[m]);
                            acc = __fadd_rn(acc, term(fx[e + 1], mask & 2, pc, p[m + 2]));
                            acc = __fadd_rn(acc, term(fy[e], mask & 4, pc, lo_j[m * 256]));
                            acc = __fadd_rn(acc, term(fy[2 + e], mask & 8, pc, hi_j[m * 256]));
                            acc = __fadd_rn(acc, term(fz[e], mask & 16, pc, lo_k[m * 256]));
                            acc = __fadd_rn(acc, term(fz[2 + e], mask & 32, pc, hi_k[m * 256]));
                            a[m] = mask & 64 ? pc : __fadd_rn(pc, __fmul_rn(c_dt, acc));
                        }
                        asm volatile("" ::: "memory");
                    }
                } else if (T.unit) {
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const float pc = p[m + 1];
                        float acc = __fadd_rn(__fsub_rn(pc, p[m]), __fsub_rn(pc, p[m + 2]));
                        acc = __fadd_rn(acc, __fsub_rn(pc, lo_j[m * 256]));
                        acc = __fadd_rn(acc, __fsub_rn(pc, hi_j[m * 256]));
                        acc = __fadd_rn(acc, __fsub_rn(pc, lo_k[m * 256]));
                        a[m] = __fadd_rn(acc, __fsub_rn(pc, hi_k[m * 256]));
                    }
                } else if (!kLattice || T.face >= 0) {
                    const float* fx = sm + T.face + lt;
                    const float* fy = sm + T.face + kBoxY + lt;
                    const float* fz = sm + T.face + kBoxZ + row * 33 + lane;
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const float pc = p[m + 1];
                        float acc = __fmul_rn(fx[m * 256], __fsub_rn(pc, p[m]));
                        acc = __fadd_rn(acc, __fmul_rn(fx[m * 256 + 256], __fsub_rn(pc, p[m + 2])));
                        acc = __fadd_rn(acc, __fmul_rn(fy[m * 288], __fsub_rn(pc, lo_j[m * 256])));
                        acc = __fadd_rn(acc, __fmul_rn(fy[m * 288 + 32], __fsub_rn(pc, hi_j[m * 256])));
                        acc = __fadd_rn(acc, __fmul_rn(fz[m * 264], __fsub_rn(pc, lo_k[m * 256])));
                        a[m] = __fadd_rn(acc, __fmul_rn(fz[m * 264 + 1], __fsub_rn(pc, hi_k[m * 256])));
                    }
                } else {
                    // no box left: the fractions from the lattices
                    const int j = T.j0 + row, k = T.k0 + lane;
#pragma unroll
                    for (int m0 = 0; m0 < 4; m0 += 2) {
                        float fx[3], fy[4], fz[4];
                        coefficients(T.i0 + m0, j, k, fx, fy, fz);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int m = m0 + e;
                            const float pc = p[m + 1];
                            float acc = __fmul_rn(fx[e], __fsub_rn(pc, p[m]));
                            acc = __fadd_rn(acc, __fmul_rn(fx[e + 1], __fsub_rn(pc, p[m + 2])));
                            acc = __fadd_rn(acc, __fmul_rn(fy[e], __fsub_rn(pc, lo_j[m * 256])));
                            acc = __fadd_rn(acc, __fmul_rn(fy[2 + e], __fsub_rn(pc, hi_j[m * 256])));
                            acc = __fadd_rn(acc, __fmul_rn(fz[e], __fsub_rn(pc, lo_k[m * 256])));
                            a[m] = __fadd_rn(acc, __fmul_rn(fz[2 + e], __fsub_rn(pc, hi_k[m * 256])));
                        }
                        asm volatile("" ::: "memory");
                    }
                }
                if (!HEAT) div_rn4(a, hhd);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    ap[s * 4 + m] = a[m];
                    pAp[s] = __fma_rn((double)p[m + 1], (double)a[m], pAp[s]);   // the product of two floats is exact
                }
                if (kWide) {
                    int cells;
                    const int t = first_cell(T, cells);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (m < cells) S.cg_Ap[t + m * nn] = a[m];
                    stash(q, pAp);
                }
            }
            if (!kWide) stash(g, pAp);
            ok = exchange<1, NT>(team, nt, step, red, tsum, sums, bad, [] {}, [&](const double (&tot)[1]) {
                Ls.pAp = tot[0];
                Ls.alpha = __double2float_rn(quotient(Ls.rz, tot[0]));
            });
            if (!ok) break;
            const float alpha = Ls.alpha;
            // x += alpha p, r -= alpha A p, z = D r; z of the shared faces goes out; r.r and r.z
            double part[2 * QR];
            ++pub;
#pragma unroll (kWide ? 2 : QR)
            for (int turn = 0; turn < turns; ++turn) {
                const int s = kWide ? 0 : turn, q = G * turn + g;
                part[s] = part[QR + s] = 0.0;
                if (q >= nt) continue;
                float d[4], z4[4];
                diag(tt[q], s, d);
                const float* core = sm + q * 1024 + lt;
                float* x = sm + X + q * 1024 + lt;
                if constexpr (kWide) {
                    int cells;
                    const int t = first_cell(tt[q], cells);
                    float xv[4];
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const bool in = m < cells;
                        r[m] = in ? S.cg_r[t + m * nn] : 0.0f;
                        ap[m] = in ? S.cg_Ap[t + m * nn] : 0.0f;
                        xv[m] = in ? xg[t + m * nn] : 0.0f;
                    }
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        r[m] = __fsub_rn(r[m], __fmul_rn(alpha, ap[m]));
                        if (m < cells) {
                            S.cg_r[t + m * nn] = r[m];
                            xg[t + m * nn] = __fadd_rn(xv[m], __fmul_rn(alpha, core[m * 256]));
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int e = s * 4 + m;
                    if (kKeepX)
                        xr[e] = __fadd_rn(xr[e], __fmul_rn(alpha, pr[e]));
                    else if (!kWide)
                        x[m * 256] = __fadd_rn(x[m * 256], __fmul_rn(alpha, core[m * 256]));
                    if (!kWide) r[e] = __fsub_rn(r[e], __fmul_rn(alpha, ap[e]));
                    z4[m] = __fmul_rn(d[m], r[e]);
                    part[s] = __fma_rn((double)r[e], (double)r[e], part[s]);
                    part[QR + s] = __fma_rn((double)r[e], (double)z4[m], part[QR + s]);
                }
                post(tt[q], z4, team.base | (pub & 0x3ffu));
                if (kWide) stash(q, part);
            }
            if (!kWide) stash(g, part);
            {
                ok = exchange<2, NT>(team, nt, step, red, tsum, sums, bad, [&] { fetch(team.base | (pub & 0x3ffu)); },
                                     [&](const double (&tot)[2]) {
                                         // the classic test, then beta (update_scalars)
                                         const double rr = tot[0];
                                         const bool above = rr > Ls.atol_sq, finite = isfinite(rr);
                                         Ls.beta = above ? __double2float_rn(quotient(tot[1], Ls.rz)) : 0.0f;
                                         Ls.rz = tot[1];
                                         Ls.rr = rr;
                                         Ls.iters = kit;
                                         if (!finite) Ls.status |= HF_SCENE_NONFINITE;
                                         Ls.live = above && finite && kit < Ls.maxit;
                                         if (!Ls.live && above && finite) Ls.status |= HEAT ? HF_SCENE_HEAT_MAXITER : HF_SCENE_PRESSURE_MAXITER;
                                     });
                if (!ok) break;
                beta = Ls.beta;
                live = Ls.live;
            }
        }
        // ------------------------------------------------------------- heat: x back
        if (HEAT && !kWide && ok) {
#pragma unroll QR
            for (int turn = 0; turn < turns; ++turn) {
                const int q = G * turn + g;
                if (q >= nt) continue;
                int cells;
                const int t = first_cell(tt[q], cells);
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (m < cells) xg[t + m * nn] = kKeepX ? xr[turn * 4 + m] : sm[X + q * 1024 + m * 256 + lt];
            }
        }
        // ------------------------------------------------------------- pressure: x back, projection (grid.py:140-153)
        if (!HEAT && ok) {
            ++pub;
#pragma unroll QR
            for (int turn = 0; turn < turns; ++turn) {
                const int s = kWide ? 0 : turn, q = G * turn + g;
                if (q >= nt) continue;
                float x4[4];
                int cells;
                const int t = first_cell(tt[q], cells);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    float& x = sm[X + q * 1024 + m * 256 + lt];
                    if (kKeepX) x = xr[s * 4 + m];
                    if (kWide) x = m < cells ? S.p[t + m * nn] : 0.0f;
                    x4[m] = x;
                }
                if ((int)blockIdx.x != c_absent_block - kAbsentLate) post(tt[q], x4, team.base | (pub & 0x3ffu));
            }
            __syncthreads();
            if (warp >= kPollWarps) fetch(team.base | (pub & 0x3ffu));
            take(team.base | (pub & 0x3ffu), [&](float& pb, float v) { pb = v; });
            ok = !__syncthreads_or(bad);
        }
        if (!HEAT && ok) {
            float *u = S.u[par ^ 1], *v = S.v[par ^ 1], *w = S.w[par ^ 1];
            const float dtr = (float)(dt_d / S.rho);
            const DivBy hd = div_by(h);
            for (int q = g; q < nt; q += G) {
                const BrickTile& T = tt[q];
                auto at = [&](int o) { return o < X ? o + X : o; };   // the x of another tile of the block, or the halo
                const int core = X + q * 1024 + lt, j = T.j0 + row, k = T.k0 + lane;
                const float* lo_j = sm + (row == 0 ? at(T.nb[2]) + lane : core - 32);
                const float* lo_k = sm + (lane == 0 ? at(T.nb[4]) + row * 32 : core - 1);
                int cells;
                const int t = first_cell(T, cells), fv = vidx_(n, T.i0, j, k), fw = widx_(n, T.i0, j, k);
                // the tile's faces are requested together
                float x[5], du[4], dv[4], dw[4], uo[4], vo[4], wo[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const bool in = m < cells;
                    uo[m] = in ? u[t + m * nn] : 0.0f;
                    vo[m] = in ? v[fv + m * (nn + n)] : 0.0f;
                    wo[m] = in ? w[fw + m * (nn + n)] : 0.0f;
                }
                x[0] = sm[at(T.nb[0]) + lt];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    x[m + 1] = sm[core + m * 256];
                    du[m] = __fmul_rn(dtr, __fsub_rn(x[m + 1], x[m]));
                    dv[m] = __fmul_rn(dtr, __fsub_rn(x[m + 1], lo_j[m * 256]));
                    dw[m] = __fmul_rn(dtr, __fsub_rn(x[m + 1], lo_k[m * 256]));
                }
                div_rn4(du, hd);
                div_rn4(dv, hd);
                div_rn4(dw, hd);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    if (m >= cells) continue;
                    const int i = T.i0 + m;
                    if (!kWide) S.p[t + m * nn] = x[m + 1];
                    u[t + m * nn] = i == 0 ? 0.0f : __fsub_rn(uo[m], du[m]);
                    v[fv + m * (nn + n)] = j == 0 ? 0.0f : __fsub_rn(vo[m], dv[m]);
                    w[fw + m * (nn + n)] = k == 0 ? 0.0f : __fsub_rn(wo[m], dw[m]);
                    if (i == n - 1) u[uidx_(n, n, j, k)] = 0.0f;
                    if (j == n - 1) v[vidx_(n, i, n, k)] = 0.0f;
                    if (k == n - 1) w[widx_(n, i, j, n)] = 0.0f;
                }
            }
        }
        __syncthreads();
        if (!ok) {
            // The first block reports the scene, and it may have finished where this one gave up: the last block to leave the
            // launch then takes that back (below).
            if (threadIdx.x == 0) {
                s_gave_up = 1;
                atomicOr(ws.arrive + job, kGaveUp | (par ? kParity : 0u));
            }
        }
        if (bl.jobs > 1 && threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ws.arrive + job) : "memory");
            left = job;
            left_nb = J.z;
        }
        if (leader && threadIdx.x == 0) write_stats(S, Ls, HEAT, !ok, par);
        __syncthreads();
    }
    // the last block to leave prepares the next launch: another launch number, no error, no arrivals
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned before = atomicAdd(ws.brick + 1, s_gave_up ? 0x10001u : 1u);   // low half: blocks; high: those that gave up
        if ((before & 0xffffu) == gridDim.x - 1) {
            const bool any = s_gave_up || before >> 16;
            if (any) take_back(scenes, ws.arrive, ws.jobs, bl.jobs, bl.job0.x, HEAT);
            if (bl.jobs > 1 || any)
                for (int q = 0; q < bl.jobs; ++q) ws.arrive[q] = 0;
            ws.brick[1] = 0;
            ws.brick[2] = 0;
            ws.brick[0] = launch + 1;
        }
    }
}

// quotient, elementwise (checked against the operator)
__global__ void k_quotient(int count, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) out[i] = quotient(a[i], b[i]);
}

template <bool HEAT>
static const void* pick(int tiles) {
    if (tiles <= 2) return (const void*)k_brick<2, 1, HEAT>;
    if (tiles <= 4) return (const void*)k_brick<4, 1, HEAT>;
    if (tiles <= 6) return (const void*)k_brick<3, 2, HEAT>;
    if (tiles <= 9) return (const void*)k_brick<3, 3, HEAT>;
    if (tiles <= kBrickMaxTiles) return (const void*)k_brick<3, 5, HEAT>;
    return (const void*)k_brick<3, 0, HEAT>;
}

const void* brick_kernel(const BrickLaunch& bl, bool heat, int* threads) {
    // the small pressure variants keep every tile's fractions in a box (launch_brick passes fewer where they do not fit)
    const int tiles = !heat && bl.boxes < bl.tiles && bl.tiles <= kBrickMaxTiles ? kBrickMaxTiles : bl.tiles;
    *threads = tiles <= 2 ? 512 : tiles <= 4 ? 1024 : 768;
    return heat ? pick<true>(tiles) : pick<false>(tiles);
}

size_t brick_smem(const BrickLaunch& bl) {
    const size_t per_tile = bl.tiles <= kBrickMaxTiles ? 2048 : 1024;
    return (bl.tiles * per_tile + (size_t)bl.pages * 1024 + (size_t)bl.boxes * kFaceBox) * sizeof(float);
}

int brick_box_bytes() { return kFaceBox * (int)sizeof(float); }

int brick_set_wait_limit(unsigned long long limit_ns, int absent_block) {
    if (cudaMemcpyToSymbol(c_wait_limit_ns, &limit_ns, sizeof limit_ns) != cudaSuccess) return HF_ERR_CUDA;
    if (cudaMemcpyToSymbol(c_absent_block, &absent_block, sizeof absent_block) != cudaSuccess) return HF_ERR_CUDA;
    return HF_OK;
}

}  // namespace hf
