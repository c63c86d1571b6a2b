// hf_api.cu -- host side of the C ABI declared in include/heatflow_b200.h.
//
// Stateless apart from a per-device cache of SM count and cooperative-launch occupancies.  No function allocates device
// memory; the workspace layout below carves the caller's buffer (barrier counters, offset tables, the scenes' TMA
// descriptors, the CG partial sums).
#include <algorithm>
#include <cstdio>
#include <cudaTypedefs.h>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "hf_cg.cuh"

namespace {

thread_local std::string g_err;

int fail(int code, const char* what, cudaError_t e = cudaSuccess) {
    char buf[512];
    if (e != cudaSuccess)
        std::snprintf(buf, sizeof buf, "%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
    else
        std::snprintf(buf, sizeof buf, "%s", what);
    g_err = buf;
    return code;
}

#define HF_CUDA(call, what)                                  \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return fail(HF_ERR_CUDA, what, e_); \
    } while (0)

struct DeviceInfo {
    int sms = 0;
    int coop = 0;
    int occ_heat = 0, occ_pressure = 0, occ_pressure_tma = 0;
    size_t smem_optin = 0;
    bool ready = false;
    bool brick_ready[3][hf::kBrickWideTiles + 1];  // the on-chip pressure solve's kernels whose shared-memory limit is raised
};

std::mutex g_mu;
DeviceInfo g_dev[64];

int device_info(DeviceInfo** out) {
    int dev = 0;
    HF_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= 64) return fail(HF_ERR_DEVICE, "device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_mu);
    DeviceInfo& d = g_dev[dev];
    if (!d.ready) {
        int major = 0;
        HF_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev), "cudaDeviceGetAttribute");
        if (major != 10) return fail(HF_ERR_DEVICE, "libheatflow_b200 is built for sm_100a (B200); this device is not sm_100");
        HF_CUDA(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
        HF_CUDA(cudaDeviceGetAttribute(&d.coop, cudaDevAttrCooperativeLaunch, dev), "cudaDeviceGetAttribute");
        HF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.occ_heat, hf::pcg_kernel(true, false), hf::kThreads, 0),
                "occupancy");
        HF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.occ_pressure, hf::pcg_kernel(false, false), hf::kThreads, 0),
                "occupancy");
        HF_CUDA(cudaFuncSetAttribute(hf::pcg_kernel(false, true), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)hf::pcg_stream_smem(true)),
                "smem attribute (streaming CG)");
        HF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.occ_pressure_tma, hf::pcg_kernel(false, true), hf::kThreads,
                                                              hf::pcg_stream_smem(true)),
                "occupancy");
        HF_CUDA(cudaFuncSetAttribute(hf::k_face_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hf::face_tile_smem()),
                "smem attribute (face stage)");
        HF_CUDA(cudaFuncSetAttribute(hf::k_advect_T_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)hf::advect_tile_smem()),
                "smem attribute (temperature stage)");
        int optin = 0;
        HF_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "cudaDeviceGetAttribute");
        d.smem_optin = (size_t)optin;
        if (!d.coop) return fail(HF_ERR_DEVICE, "device does not support cooperative launches");
        std::memset(d.brick_ready, 0, sizeof d.brick_ready);
        d.ready = true;
    }
    *out = &d;
    return HF_OK;
}

constexpr long long kGroupCells = 2400000;   // cells of one CG group by default (one 128^3 or two 96^3 scenes)
constexpr size_t kHeadBytes = 256;           // barrier counters, group queue, lane slots, timeout flag

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct Layout {
    size_t head, chunk_begin, tile_begin, maps, partA, partB, mean_part, streaming;   // streaming: bytes of a plan that only streams
    size_t brick, arrive, jobs, mail, halo, total;
};

Layout layout(int S, int C, int T) {
    Layout L{};
    size_t o = 0;
    L.head = o;                      // bar[2 kMaxLanes], queue[2], lane_next[2 kMaxLanes], err -> 256 bytes
    o = align_up(o + kHeadBytes, 256);
    L.chunk_begin = o;
    o = align_up(o + sizeof(int) * (size_t)(S + 1), 256);
    L.tile_begin = o;
    o = align_up(o + sizeof(int) * (size_t)(S + 1), 256);
    L.maps = o;                      // kMapsPerScene TMA descriptors per scene (128 bytes each)
    o = align_up(o + sizeof(CUtensorMap) * hf::kMapsPerScene * (size_t)S, 256);
    L.partA = o;                     // 3 doubles per tile, component-major
    o = align_up(o + sizeof(double) * 3 * (size_t)T, 256);
    L.partB = o;
    o = align_up(o + sizeof(double) * 3 * (size_t)T, 256);
    L.mean_part = o;
    o = align_up(o + sizeof(double) * (size_t)C, 256);
    L.streaming = o;
    // A plan of more tiles than its scenes can have on the chip streams: nothing below is used, nor sized for the rest of them
    // (not left out, so that a plan whose large scenes are inactive at upload still fits).
    T = (int)std::min<long long>(T, (long long)S * hf::kUnits * hf::kBrickWideTiles);
    L.brick = o;                     // the on-chip solve: launch, leave and error words
    o = align_up(o + 256, 256);
    L.arrive = o;
    o = align_up(o + sizeof(unsigned) * (size_t)S, 256);
    L.jobs = o;
    o = align_up(o + sizeof(int4) * (size_t)S, 256);
    L.mail = o;                      // a line per unit of a block (one per tile at most), two parities, min(T, kUnits) blocks at most
    o = align_up(o + 128u * 2u * hf::kBrickWideTiles * (size_t)hf::unit_count(T), 256);
    L.halo = o;
    o = align_up(o + sizeof(unsigned long long) * hf::kHaloEntries * (size_t)T, 256);
    L.total = o;
    return L;
}

hf::Workspace workspace(const hf_plan* p) {
    const Layout L = layout(p->num_scenes, p->num_chunks, p->num_tiles);
    char* b = static_cast<char*>(p->workspace);
    hf::Workspace w;
    w.bar = reinterpret_cast<unsigned*>(b + L.head);
    w.queue = w.bar + 2 * hf::kMaxLanes;
    w.lane_next = reinterpret_cast<int*>(w.queue + 2);
    w.err = w.lane_next + 2 * hf::kMaxLanes;
    w.chunk_begin = reinterpret_cast<int*>(b + L.chunk_begin);
    w.tile_begin = reinterpret_cast<int*>(b + L.tile_begin);
    w.maps = reinterpret_cast<const CUtensorMap*>(b + L.maps);
    w.partA = reinterpret_cast<double*>(b + L.partA);
    w.partB = reinterpret_cast<double*>(b + L.partB);
    w.mean_part = reinterpret_cast<double*>(b + L.mean_part);
    w.brick = reinterpret_cast<unsigned*>(b + L.brick);
    w.arrive = reinterpret_cast<unsigned*>(b + L.arrive);
    w.jobs = reinterpret_cast<int4*>(b + L.jobs);
    w.mail = reinterpret_cast<ulonglong2*>(b + L.mail);
    w.halo = reinterpret_cast<unsigned long long*>(b + L.halo);
    w.tiles = p->num_tiles;
    return w;
}

int tiles_of(int n) { return ((n + hf::kTI - 1) / hf::kTI) * ((n + hf::kTJ - 1) / hf::kTJ) * ((n + hf::kTK - 1) / hf::kTK); }

// TMA descriptor of a 3-D float array (k fastest) of dims (nk, nj, ni) with a box (bk, bj, bi)
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

int encode_map(CUtensorMap* m, const float* base, int nk, int nj, int ni, int bk, int bj, int bi) {
    if (!g_encode) {
        cudaDriverEntryPointQueryResult q;
        HF_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", reinterpret_cast<void**>(&g_encode), cudaEnableDefault, &q),
                "cudaGetDriverEntryPoint(cuTensorMapEncodeTiled)");
        if (q != cudaDriverEntryPointSuccess || !g_encode) return fail(HF_ERR_DEVICE, "cuTensorMapEncodeTiled unavailable");
    }
    const cuuint64_t dims[3] = {(cuuint64_t)nk, (cuuint64_t)nj, (cuuint64_t)ni};
    const cuuint64_t strides[2] = {(cuuint64_t)nk * 4u, (cuuint64_t)nk * nj * 4u};
    const cuuint32_t box[3] = {(cuuint32_t)bk, (cuuint32_t)bj, (cuuint32_t)bi};
    const cuuint32_t es[3] = {1, 1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(HF_ERR_DEVICE, "cuTensorMapEncodeTiled failed");
    return HF_OK;
}

// The six TMA descriptors of a scene's tiled pressure stencil: z and both search-direction buffers with a one-cell halo,
// alpha_f x on its face lattice, alpha_f y and z in cell layout.
int encode_scene_maps(const hf_scene& sc, CUtensorMap* m) {
    const int n = sc.n;
    int rc;
    if ((rc = encode_map(&m[0], sc.cg_z, n, n, n, 40, 10, 6))) return rc;
    if ((rc = encode_map(&m[1], sc.cg_p[0], n, n, n, 40, 10, 6))) return rc;
    if ((rc = encode_map(&m[2], sc.cg_p[1], n, n, n, 40, 10, 6))) return rc;
    if ((rc = encode_map(&m[3], sc.ax, n, n, n + 1, 32, 8, 5))) return rc;
    if ((rc = encode_map(&m[4], sc.ayc, n, n, n, 32, 9, 4))) return rc;
    return encode_map(&m[5], sc.azc, n, n, n, 36, 8, 4);
}

int check_plan(const hf_plan* p) {
    if (!p || !p->scenes_host || !p->scenes_dev || !p->work_dev || !p->workspace) return fail(HF_ERR_ARG, "incomplete hf_plan");
    if (p->num_scenes <= 0 || p->num_scenes > hf::kMaxScenes) return fail(HF_ERR_ARG, "num_scenes out of range (1..1024)");
    if (!p->tiles_dev) return fail(HF_ERR_ARG, "incomplete hf_plan (tile table)");
    if (p->workspace_bytes < layout(p->num_scenes, p->num_chunks, p->num_tiles).streaming)
        return fail(HF_ERR_WORKSPACE, "workspace smaller than hf_workspace_bytes()");
    return HF_OK;
}

inline cudaStream_t S(void* s) { return static_cast<cudaStream_t>(s); }

bool any_flag(const hf_plan* p, unsigned f) {
    for (int s = 0; s < p->num_scenes; ++s)
        if ((p->scenes_host[s].flags & HF_FLAG_ACTIVE) && (p->scenes_host[s].flags & f)) return true;
    return false;
}

// How the on-chip solves share the blocks among a plan's active scenes: a team of blocks for each (brick_teams, which every
// launch forms again: a few us for 64 scenes), and the places of the teams in the blocks' common order (brick_jobs, once at
// the upload).
struct BrickTeam {
    int scene, n, T, blocks, most;   // most: tiles that one of the blocks owns
};
// teams, blocks of the launch, the most tiles that a block owns and the most tiles along k of a scene
struct BrickSchedule {
    int jobs, blocks, tiles, tk;
};

// the most tiles of a block when `blocks` blocks share a scene of T tiles in whole units (hf_brick.cu)
int brick_tiles(int T, int blocks) {
    const int units = hf::unit_count(T);
    int most = 0;
    for (int b = 0, first = 0; b < blocks; ++b) {
        const int end = hf::unit_first(T, units, units * (b + 1) / blocks);
        most = std::max(most, end - first);
        first = end;
    }
    return most;
}

// False when a scene does not fit: with `cap` kBrickMaxTiles, 148 blocks hold 2220 tiles (an edge of 128 has 2048), with
// kBrickWideTiles 5328 (an edge of 168 has 5292).
// Scenes that fit side by side share the blocks in proportion to their tiles.  Otherwise each gets as few blocks as hold
// it: the more tiles a block has, the less its reductions weigh.  team: room for kMaxScenes.
bool brick_teams(const hf_plan* p, int sms, int cap, BrickTeam* team, BrickSchedule& out) {
    const int blocks = std::min(sms, hf::kUnits);
    out = BrickSchedule{0, blocks, 0, 0};
    // the fewest blocks that hold a scene of edge n, and their most tiles: found once for each edge (the divisions of a
    // search take a few us)
    struct Fit {
        int blocks, most;
    } fits[hf::kBrickEdge + 1] = {};
    int least = 0;
    for (int s = 0; s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        if (!(sc.flags & HF_FLAG_ACTIVE)) continue;
        if (sc.n < 2 || sc.n > hf::kBrickEdge) return false;
        const int T = tiles_of(sc.n);
        Fit& fit = fits[sc.n];
        if (!fit.blocks) {
            fit.blocks = (T + cap - 1) / cap;
            while (fit.blocks <= std::min(blocks, T) && (fit.most = brick_tiles(T, fit.blocks)) > cap) ++fit.blocks;
            if (fit.blocks > std::min(blocks, T)) return false;
        }
        team[out.jobs++] = BrickTeam{s, sc.n, T, fit.blocks, fit.most};
        least += fit.blocks;
        out.tk = std::max(out.tk, (sc.n + hf::kTK - 1) / hf::kTK);
    }
    if (!out.jobs) return false;
    if (least <= blocks) {
        // side by side: the blocks that are left go, one at a time, to the scene whose blocks own the most tiles
        for (; least < blocks; ++least) {
            BrickTeam* most = nullptr;
            for (BrickTeam* w = team; w < team + out.jobs; ++w)
                if (w->blocks < std::min(blocks, w->T) && (!most || (long long)w->T * most->blocks > (long long)most->T * w->blocks)) most = w;
            if (!most) break;
            ++most->blocks;
        }
        out.blocks = least;
        for (int q = 0; q < out.jobs; ++q) team[q].most = brick_tiles(team[q].T, team[q].blocks);
    }
    for (int q = 0; q < out.jobs; ++q) out.tiles = std::max(out.tiles, team[q].most);
    return true;
}

bool brick_teams(const hf_plan* p, int sms, BrickTeam* team, BrickSchedule& out) {
    return brick_teams(p, sms, hf::kBrickMaxTiles, team, out) || brick_teams(p, sms, hf::kBrickWideTiles, team, out);
}

// The jobs (scene, first block, blocks, the most tiles of a block): the largest scenes come first, each on the contiguous
// blocks that are free the soonest.
std::vector<int4> brick_jobs(const BrickTeam* team, const BrickSchedule& sched) {
    std::vector<BrickTeam> order(team, team + sched.jobs);
    std::stable_sort(order.begin(), order.end(), [](const BrickTeam& a, const BrickTeam& b) { return a.T > b.T; });
    std::vector<double> until(sched.blocks, 0.0);
    std::vector<int> high(sched.blocks);   // blocks of the window, each busy for longer than all after it
    std::vector<int4> jobs;
    for (const BrickTeam& w : order) {
        int at = 0, head = 0, tail = 0;
        double best = 0.0;
        for (int e = 0; e < sched.blocks; ++e) {   // the window's last block
            while (tail > head && until[high[tail - 1]] <= until[e]) --tail;
            high[tail++] = e;
            const int f = e - w.blocks + 1;
            if (f < 0) continue;
            if (high[head] < f) ++head;
            const double t = until[high[head]];
            if (f == 0 || t < best) {
                best = t;
                at = f;
            }
        }
        // an iteration takes about 1.6 us of exchanges and 0.35 us a tile; iterations grow like the edge
        std::fill(until.begin() + at, until.begin() + at + w.blocks, best + w.n * (1.6 + 0.35 * w.most));
        jobs.push_back(make_int4(w.scene, at, w.blocks, w.most));
    }
    return jobs;
}

// The on-chip solve of a plan whose scenes all fit.  HF_OK after launching, -1 when it does not apply.
int launch_brick(const hf_plan* p, DeviceInfo* d, bool heat, double dt, void* stream) {
    if (!(p->options & HF_PLAN_MAPS_READY) || p->workspace_bytes < layout(p->num_scenes, p->num_chunks, p->num_tiles).total) return -1;
    static thread_local BrickTeam team[hf::kMaxScenes];
    BrickSchedule sched;
    if (!brick_teams(p, d->sms, team, sched)) return -1;
    for (int s = 0; s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        if ((sc.flags & HF_FLAG_ACTIVE) && (!sc.pdiag || !sc.hdiag || !sc.cg_r || !sc.cg_z || !sc.cg_Ap)) return -1;   // scratch of the larger variants
    }
    hf::BrickLaunch bl;
    std::memset(&bl, 0, sizeof bl);
    bl.jobs = sched.jobs;
    bl.job0 = make_int4(team[0].scene, 0, team[0].blocks, sched.tiles);   // of several jobs the places are in the workspace
    bl.tiles = sched.tiles;
    // A block's run of tiles is contiguous in (k, i, j): at most 2 tk of its i faces, all of its j faces and the two k
    // faces at the run's ends border other blocks.
    bl.i_pages = (2 * std::min(sched.tk, bl.tiles) + 3) / 4;
    bl.j_pages = (2 * bl.tiles + 7) / 8;
    bl.pages = bl.i_pages + bl.j_pages + 1;
    // as many boxes of face fractions as fit beside the rest and the kernel's own arrays (up to 8 and 18 KB); further
    // general tiles read the lattices
    const size_t room = d->smem_optin - (bl.tiles <= hf::kBrickMaxTiles ? 9 : 19) * 1024, base = hf::brick_smem(bl);
    if (base > room) return -1;
    bl.boxes = heat ? 0 : std::min(bl.tiles, (int)((room - base) / hf::brick_box_bytes()));
    int threads = 0;
    const void* fn = hf::brick_kernel(bl, heat, &threads);
    bool& ready = d->brick_ready[heat ? 2 : bl.boxes < bl.tiles][bl.tiles];
    if (!ready) {
        cudaFuncAttributes at;
        HF_CUDA(cudaFuncGetAttributes(&at, fn), "attributes (on-chip CG)");
        HF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(d->smem_optin - at.sharedSizeBytes)),
                "smem attribute (on-chip CG)");
        ready = true;
    }
    hf::Workspace ws = workspace(p);
    const hf_scene* scenes = static_cast<const hf_scene*>(p->scenes_dev);
    const hf::TileItem* tiles = static_cast<const hf::TileItem*>(p->tiles_dev);
    void* args[] = {(void*)&scenes, (void*)&tiles, (void*)&dt, (void*)&ws, (void*)&bl};
    HF_CUDA(cudaLaunchCooperativeKernel(fn, dim3(sched.blocks), dim3(threads), args, hf::brick_smem(bl), S(stream)),
            "cooperative launch (on-chip CG)");
    return HF_OK;
}

// Both CG solves of a plan.  The on-chip solve where every active scene fits it.  Otherwise one launch of the
// streaming kernel: the active scenes are cut, in table order, into groups of at most kGroupScenes scenes and
// group_cells cells (default kGroupCells: a group's CG vectors stay in L2), solved by the lanes of the grid.
int launch_pcg(const hf_plan* p, bool heat, double dt, void* stream) {
    DeviceInfo* d = nullptr;
    int rc = device_info(&d);
    if (rc) return rc;
    if (p->num_tiles == 0) return HF_OK;
    int nactive = 0, total = 0;
    bool correction = false;   // the outer defect correction runs in the streaming kernel only
    for (int s = 0; s < p->num_scenes; ++s)
        if (p->scenes_host[s].flags & HF_FLAG_ACTIVE) {
            ++nactive;
            total += tiles_of(p->scenes_host[s].n);
            correction = correction || (p->scenes_host[s].flags & HF_FLAG_DEFECT_CORRECTION);
        }
    if (total != p->num_tiles) return fail(HF_ERR_ARG, "plan changed since hf_plan_upload");
    if (nactive > 0 && !correction && !(p->options & HF_PLAN_STREAMING_CG) &&
        !(heat && nactive == 1 && (p->options & HF_PLAN_STREAMING_HEAT))) {
        rc = launch_brick(p, d, heat, dt, stream);
        if (rc != -1) return rc;
    }
    static thread_local hf::GroupTable gt;   // 16 KB: kept off the stack; the launch copies it
    gt.count = 0;
    const long long budget = p->group_cells > 0 ? p->group_cells : kGroupCells;
    int s_lo = -1, s_last = -1, t_lo = 0, t = 0;
    long long cells = 0;
    for (int s = 0; s <= p->num_scenes; ++s) {
        const bool end = s == p->num_scenes;
        if (!end && !(p->scenes_host[s].flags & HF_FLAG_ACTIVE)) continue;
        const long long c = end ? 0 : (long long)p->scenes_host[s].n * p->scenes_host[s].n * p->scenes_host[s].n;
        if (s_lo >= 0 && (end || cells + c > budget || s + 1 - s_lo > hf::kGroupScenes)) {
            // the group ends after its last active scene: [s_lo, s_last] spans at most kGroupScenes scenes
            if (gt.count == hf::kMaxGroups) return fail(HF_ERR_ARG, "more CG groups than one launch takes");
            gt.g[gt.count++] = make_int4(s_lo, s_last + 1, t_lo, t);
            s_lo = -1;
        }
        if (end) break;
        if (s_lo < 0) {
            s_lo = s;
            t_lo = t;
            cells = 0;
        }
        cells += c;
        s_last = s;
        t += tiles_of(p->scenes_host[s].n);
    }
    // the pressure stencil from TMA-staged boxes when the plan's descriptors exist and every active scene has them
    bool tma = !heat && (p->options & HF_PLAN_MAPS_READY) && !(p->options & HF_PLAN_NO_TMA);
    for (int s = 0; tma && s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        // the same test as hf_plan_upload's: only then does the workspace hold this scene's descriptors
        if ((sc.flags & HF_FLAG_ACTIVE) && (sc.n % 4 != 0 || !sc.cg_z || !sc.cg_p[0] || !sc.cg_p[1] || !sc.ax || !sc.ayc ||
                                            !sc.azc || !sc.p || !sc.cg_r || !sc.cg_Ap || !sc.pdiag))
            tma = false;
    }
    const int occ = heat ? d->occ_heat : tma ? d->occ_pressure_tma : d->occ_pressure;
    if (occ <= 0) return fail(HF_ERR_DEVICE, "persistent CG kernel does not fit on an SM");
    int lanes = (int)((p->options >> HF_PLAN_LANES_SHIFT) & 15u);
    if (lanes <= 0) lanes = 1;
    if (lanes > hf::kMaxLanes) lanes = hf::kMaxLanes;
    if (lanes > gt.count) lanes = gt.count;
    int grid = p->persistent_blocks > 0 ? p->persistent_blocks : d->sms * (occ < 2 ? occ : 2);
    if (grid > d->sms * occ) grid = d->sms * occ;
    grid -= grid % lanes;
    if (grid < lanes) grid = lanes;
    gt.lanes = lanes;
    hf::Workspace ws = workspace(p);
    const hf_scene* scenes = static_cast<const hf_scene*>(p->scenes_dev);
    const hf::TileItem* tiles = static_cast<const hf::TileItem*>(p->tiles_dev);
    HF_CUDA(cudaMemsetAsync(ws.bar, 0, kHeadBytes, S(stream)), "cudaMemsetAsync(barrier)");
    void* args[] = {(void*)&scenes, (void*)&tiles, (void*)&dt, (void*)&ws, (void*)&gt};
    HF_CUDA(cudaLaunchCooperativeKernel(hf::pcg_kernel(heat, tma), dim3(grid), dim3(hf::kThreads), args,
                                        hf::pcg_stream_smem(tma), S(stream)),
            "cooperative launch (CG)");
    return HF_OK;
}

}  // namespace

namespace hf {
size_t streaming_workspace_bytes(int num_scenes, int num_chunks, int num_tiles) {
    return layout(num_scenes, num_chunks, num_tiles).streaming;
}

int set_error(int code, const char* msg) { return fail(code, msg); }

void plan_offset_tables(const hf_plan* p, int** chunk_begin, int** tile_begin) {
    const Workspace w = workspace(p);
    *chunk_begin = w.chunk_begin;
    *tile_begin = w.tile_begin;
}
}  // namespace hf

extern "C" {

int hf_abi_version(void) { return HF_ABI_VERSION; }

const char* hf_last_error(void) { return g_err.c_str(); }

int hf_cells_per_chunk(void) { return hf::kChunk; }

int hf_chunks_for(int n) {
    if (n <= 0) return 0;
    const long long N = (long long)n * n * n;
    return (int)((N + hf::kChunk - 1) / hf::kChunk);
}

size_t hf_workspace_bytes(int num_scenes, int num_chunks, int num_tiles) {
    return layout(num_scenes, num_chunks, num_tiles).total;
}

int hf_tiles_for(int n) { return n > 0 ? tiles_of(n) : 0; }

int hf_plan_upload(hf_plan* p, void* stream) {
    if (!p || !p->scenes_host || !p->scenes_dev || !p->work_dev || !p->tiles_dev || !p->workspace)
        return fail(HF_ERR_ARG, "incomplete hf_plan");
    if (p->num_scenes <= 0 || p->num_scenes > hf::kMaxScenes) return fail(HF_ERR_ARG, "num_scenes out of range (1..1024)");
    std::vector<hf::WorkItem> work;
    std::vector<hf::TileItem> tiles;
    std::vector<int> begin(p->num_scenes + 1, 0), tbegin(p->num_scenes + 1, 0);
    for (int s = 0; s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        begin[s] = (int)work.size();
        tbegin[s] = (int)tiles.size();
        if (!(sc.flags & HF_FLAG_ACTIVE)) continue;
        if (sc.n < 2 || sc.n > 1024) return fail(HF_ERR_ARG, "scene edge n out of range (2..1024)");
        if (!sc.state) return fail(HF_ERR_ARG, "scene without a state block");
        const long long N = (long long)sc.n * sc.n * sc.n;
        for (long long f = 0; f < N; f += hf::kChunk) work.push_back(hf::WorkItem{s, (int)f});
        // k fastest, then i, then j: the six neighbours of a tile are at most (n / 32) (n / 4) tiles away in the
        // table, so tiles solved side by side share their halo rows in L2
        for (int j0 = 0; j0 < sc.n; j0 += hf::kTJ)
            for (int i0 = 0; i0 < sc.n; i0 += hf::kTI)
                for (int k0 = 0; k0 < sc.n; k0 += hf::kTK) tiles.push_back(hf::TileItem{s, i0, j0, k0});
    }
    begin[p->num_scenes] = (int)work.size();
    tbegin[p->num_scenes] = (int)tiles.size();
    p->num_chunks = (int)work.size();
    p->num_tiles = (int)tiles.size();
    const Layout L = layout(p->num_scenes, p->num_chunks, p->num_tiles);
    if (p->workspace_bytes < L.total) return fail(HF_ERR_WORKSPACE, "workspace smaller than hf_workspace_bytes()");
    HF_CUDA(cudaMemsetAsync(p->workspace, 0, L.total, S(stream)), "cudaMemsetAsync(workspace)");
    HF_CUDA(cudaMemcpyAsync(p->scenes_dev, p->scenes_host, sizeof(hf_scene) * p->num_scenes, cudaMemcpyHostToDevice, S(stream)),
            "upload scene table");
    if (!work.empty())
        HF_CUDA(cudaMemcpyAsync(p->work_dev, work.data(), sizeof(hf::WorkItem) * work.size(), cudaMemcpyHostToDevice, S(stream)),
                "upload chunk table");
    if (!tiles.empty())
        HF_CUDA(cudaMemcpyAsync(p->tiles_dev, tiles.data(), sizeof(hf::TileItem) * tiles.size(), cudaMemcpyHostToDevice, S(stream)),
                "upload tile table");
    char* b = static_cast<char*>(p->workspace);
    HF_CUDA(cudaMemcpyAsync(b + L.chunk_begin, begin.data(), sizeof(int) * begin.size(), cudaMemcpyHostToDevice, S(stream)),
            "upload chunk offsets");
    HF_CUDA(cudaMemcpyAsync(b + L.tile_begin, tbegin.data(), sizeof(int) * tbegin.size(), cudaMemcpyHostToDevice, S(stream)),
            "upload tile offsets");
    // TMA descriptors of every active scene whose stencil boxes fit the alignment rules (n % 4 == 0); zero otherwise
    std::vector<CUtensorMap> maps(hf::kMapsPerScene * (size_t)p->num_scenes);
    std::memset(maps.data(), 0, sizeof(CUtensorMap) * maps.size());
    for (int s = 0; s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        if (!(sc.flags & HF_FLAG_ACTIVE) || sc.n % 4 != 0 || !sc.cg_z || !sc.cg_p[0] || !sc.cg_p[1] || !sc.ax || !sc.ayc ||
            !sc.azc || !sc.p || !sc.cg_r || !sc.cg_Ap || !sc.pdiag)
            continue;
        CUtensorMap* m = &maps[hf::kMapsPerScene * (size_t)s];
        int rc = encode_scene_maps(sc, m);
        if (rc) return rc;
        // the CG vectors of the tile's own cells, one (32, 8, 4) box each: x (the pressure), p_0, p_1, r, Ap, D
        const float* own[6] = {sc.p, sc.cg_p[0], sc.cg_p[1], sc.cg_r, sc.cg_Ap, sc.pdiag};
        for (int q = 0; q < 6; ++q)
            if ((rc = encode_map(&m[6 + q], own[q], sc.n, sc.n, sc.n, 32, 8, 4))) return rc;
    }
    HF_CUDA(cudaMemcpyAsync(b + L.maps, maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice, S(stream)),
            "upload TMA descriptors");
    // the on-chip solves' jobs (launch_brick forms the same teams)
    std::vector<BrickTeam> team(p->num_scenes);
    std::vector<int4> jobs;
    BrickSchedule sched;
    DeviceInfo* d = nullptr;
    int drc = device_info(&d);
    if (drc) return drc;
    if (p->num_tiles && brick_teams(p, d->sms, team.data(), sched)) {
        jobs = brick_jobs(team.data(), sched);
        HF_CUDA(cudaMemcpyAsync(b + L.jobs, jobs.data(), sizeof(int4) * jobs.size(), cudaMemcpyHostToDevice, S(stream)), "upload jobs");
    }
    HF_CUDA(cudaStreamSynchronize(S(stream)), "cudaStreamSynchronize(plan upload)");
    p->options |= HF_PLAN_MAPS_READY;
    return HF_OK;
}

int hf_plan_jobs(const hf_plan* p, int sms, int* jobs) {
    if (!p || !p->scenes_host || p->num_scenes <= 0 || p->num_scenes > hf::kMaxScenes || sms < 1)
        return -fail(HF_ERR_ARG, "hf_plan_jobs: bad arguments");
    if ((p->options & HF_PLAN_STREAMING_CG) || any_flag(p, HF_FLAG_DEFECT_CORRECTION)) return 0;
    std::vector<BrickTeam> team(p->num_scenes);
    BrickSchedule sched;
    if (!brick_teams(p, sms, team.data(), sched)) return 0;
    if (jobs) std::memcpy(jobs, brick_jobs(team.data(), sched).data(), sizeof(int4) * sched.jobs);
    return sched.jobs;
}

int hf_obstacle_fields(const hf_plan* p, int all_scenes, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    const hf_scene* scenes = static_cast<const hf_scene*>(p->scenes_dev);
    const hf::WorkItem* work = static_cast<const hf::WorkItem*>(p->work_dev);
    const bool coupled = any_flag(p, HF_FLAG_PARTICLES);
    if (!coupled && !all_scenes) return HF_OK;
    for (int s = 0; s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        if (!(sc.flags & HF_FLAG_ACTIVE) || !(sc.flags & HF_FLAG_PARTICLES) || sc.n_particles <= 0) continue;
        if (!sc.acc || !sc.pos || !sc.pvel || !sc.ptemp) return fail(HF_ERR_ARG, "coupled scene without particle buffers");
        hf::k_scatter<<<(sc.n_particles + hf::kThreads - 1) / hf::kThreads, hf::kThreads, 0, S(stream)>>>(scenes, s);
    }
    if (!all_scenes) {
        // the substep's rebuild: each coupled scene over its footprint boxes only
        for (int s = 0; s < p->num_scenes; ++s) {
            const hf_scene& sc = p->scenes_host[s];
            if (!(sc.flags & HF_FLAG_ACTIVE) || !(sc.flags & HF_FLAG_PARTICLES) || sc.n_particles <= 0) continue;
            hf::k_obstacle_box<<<296, hf::kThreads, 0, S(stream)>>>(scenes, s);
        }
        for (int s = 0; s < p->num_scenes; ++s) {
            const hf_scene& sc = p->scenes_host[s];
            if (!(sc.flags & HF_FLAG_ACTIVE) || !(sc.flags & HF_FLAG_PARTICLES) || sc.n_particles <= 0) continue;
            hf::k_coeff_box<<<296, hf::kThreads, 0, S(stream)>>>(scenes, s);
        }
    } else if (p->num_chunks) {
        hf::k_obstacle<<<p->num_chunks, hf::kThreads, 0, S(stream)>>>(scenes, work, all_scenes);
        hf::k_coeff<<<p->num_chunks, hf::kThreads, 0, S(stream)>>>(scenes, work, all_scenes);
    }
    HF_CUDA(cudaGetLastError(), "launch (obstacle fields)");
    return HF_OK;
}

int hf_temperature_stage(const hf_plan* p, double dt, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    if (!p->num_chunks) return HF_OK;
    const hf_scene* scenes = static_cast<const hf_scene*>(p->scenes_dev);
    const hf::WorkItem* work = static_cast<const hf::WorkItem*>(p->work_dev);
    DeviceInfo* d = nullptr;
    if ((rc = device_info(&d))) return rc;
    hf::k_prestage<<<p->num_chunks, hf::kThreads, 0, S(stream)>>>(scenes, work, dt);
    // one 512-thread block per CG tile, the old velocities and Tw around the tile staged in shared memory
    hf::k_advect_T_tile<<<p->num_tiles, 512, hf::advect_tile_smem(), S(stream)>>>(
        scenes, static_cast<const hf::TileItem*>(p->tiles_dev), dt);
    HF_CUDA(cudaGetLastError(), "launch (temperature stage)");
    return HF_OK;
}

int hf_heat_solve(const hf_plan* p, double dt, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    return launch_pcg(p, true, dt, stream);
}

int hf_particle_update(const hf_plan* p, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    const hf_scene* scenes = static_cast<const hf_scene*>(p->scenes_dev);
    for (int s = 0; s < p->num_scenes; ++s) {
        const hf_scene& sc = p->scenes_host[s];
        if (!(sc.flags & HF_FLAG_ACTIVE) || !(sc.flags & HF_FLAG_PARTICLES) || sc.n_particles <= 0) continue;
        hf::k_particle_update<<<(sc.n_particles + hf::kThreads - 1) / hf::kThreads, hf::kThreads, 0, S(stream)>>>(scenes, s);
    }
    HF_CUDA(cudaGetLastError(), "launch (particle update)");
    return HF_OK;
}

int hf_face_stage(const hf_plan* p, double dt, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    if (!p->num_tiles) return HF_OK;
    DeviceInfo* d = nullptr;
    if ((rc = device_info(&d))) return rc;
    // one 512-thread block per CG tile, the old velocities around the tile staged in shared memory
    hf::k_face_tile<<<p->num_tiles, 512, hf::face_tile_smem(), S(stream)>>>(static_cast<const hf_scene*>(p->scenes_dev),
                                                                        static_cast<const hf::TileItem*>(p->tiles_dev), dt);
    HF_CUDA(cudaGetLastError(), "launch (face stage)");
    return HF_OK;
}

int hf_divergence_stage(const hf_plan* p, double dt, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    if (!p->num_chunks) return HF_OK;
    hf::k_divergence<<<p->num_chunks, hf::kChunk, 0, S(stream)>>>(static_cast<const hf_scene*>(p->scenes_dev),
                                                                   static_cast<const hf::WorkItem*>(p->work_dev), dt,
                                                                   workspace(p));
    HF_CUDA(cudaGetLastError(), "launch (divergence)");
    return HF_OK;
}

int hf_pressure_cg(const hf_plan* p, double dt, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    return launch_pcg(p, false, dt, stream);
}

int hf_pressure_solve(const hf_plan* p, double dt, void* stream) {
    int rc = hf_divergence_stage(p, dt, stream);
    if (rc) return rc;
    return hf_pressure_cg(p, dt, stream);
}

int hf_substep(const hf_plan* p, double dt, void* stream) {
    int rc;
    if ((rc = hf_obstacle_fields(p, 0, stream))) return rc;
    if ((rc = hf_temperature_stage(p, dt, stream))) return rc;
    if ((rc = hf_heat_solve(p, dt, stream))) return rc;
    if ((rc = hf_particle_update(p, stream))) return rc;
    if ((rc = hf_face_stage(p, dt, stream))) return rc;
    return hf_pressure_solve(p, dt, stream);
}

int hf_cell_velocity(const hf_plan* p, int s, float* out, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    if (s < 0 || s >= p->num_scenes || !out) return fail(HF_ERR_ARG, "bad scene index or output");
    hf::k_cell_velocity<<<592, 256, 0, S(stream)>>>(static_cast<const hf_scene*>(p->scenes_dev), s, out);
    HF_CUDA(cudaGetLastError(), "launch (cell velocity)");
    return HF_OK;
}

int hf_divergence_max(const hf_plan* p, int s, float* out_dev, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    if (s < 0 || s >= p->num_scenes || !out_dev) return fail(HF_ERR_ARG, "bad scene index or output");
    HF_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(float), S(stream)), "cudaMemsetAsync");
    hf::k_divergence_max<<<592, 256, 0, S(stream)>>>(static_cast<const hf_scene*>(p->scenes_dev), s,
                                                    reinterpret_cast<unsigned*>(out_dev));
    HF_CUDA(cudaGetLastError(), "launch (divergence max)");
    return HF_OK;
}

int hf_speed_max(const hf_plan* p, int s, float* out_dev, void* stream) {
    int rc = check_plan(p);
    if (rc) return rc;
    if (s < 0 || s >= p->num_scenes || !out_dev) return fail(HF_ERR_ARG, "bad scene index or output");
    HF_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(float), S(stream)), "cudaMemsetAsync");
    hf::k_speed_max<<<592, 256, 0, S(stream)>>>(static_cast<const hf_scene*>(p->scenes_dev), s,
                                               reinterpret_cast<unsigned*>(out_dev));
    HF_CUDA(cudaGetLastError(), "launch (speed max)");
    return HF_OK;
}

int hf_set_wait_limit(unsigned long long limit_ns, int absent_block) {
    if (limit_ns == 0 || limit_ns > 60000000000ull || absent_block < -1)
        return fail(HF_ERR_ARG, "hf_set_wait_limit: limit must be 1 ns .. 60 s, absent_block >= -1");
    int rc = hf::set_wait_limit(limit_ns, absent_block);
    if (rc) return fail(rc, "hf_set_wait_limit: cudaMemcpyToSymbol failed");
    return HF_OK;
}

int hf_k_divide_by(int count, const float* x, float y, float* out, void* stream) {
    if (count < 0 || (count > 0 && (!x || !out)) || !(y != 0.0f)) return fail(HF_ERR_ARG, "hf_k_divide_by: bad arguments");
    if (count == 0) return HF_OK;
    hf::k_divide_by<<<592, 256, 0, S(stream)>>>(count, x, y, out);
    HF_CUDA(cudaGetLastError(), "launch (divide_by)");
    return HF_OK;
}

int hf_k_quotient(int count, const double* a, const double* b, double* out, void* stream) {
    if (count < 0 || (count > 0 && (!a || !b || !out))) return fail(HF_ERR_ARG, "hf_k_quotient: bad arguments");
    if (count == 0) return HF_OK;
    hf::k_quotient<<<592, 256, 0, S(stream)>>>(count, a, b, out);
    HF_CUDA(cudaGetLastError(), "launch (quotient)");
    return HF_OK;
}

int hf_k_laplacian(int n, double h, double alpha, double beta, const float* p, const float* ax, const float* ay,
                   const float* az, const float* y, float* out, void* stream) {
    if (n < 1 || !p || !ax || !ay || !az || !y || !out) return fail(HF_ERR_ARG, "hf_k_laplacian: bad arguments");
    hf::k_laplacian_plain<<<592, 256, 0, S(stream)>>>(n, (float)h, (float)alpha, (float)beta, p, ax, ay, az, y, out);
    HF_CUDA(cudaGetLastError(), "launch (laplacian)");
    return HF_OK;
}

int hf_k_heat_matvec(int n, double h, double dt, double alpha, double beta, const float* x, const float* kap,
                     const uint8_t* cell_flags, const float* y, float* out, void* stream) {
    if (n < 1 || !x || !kap || !cell_flags || !y || !out) return fail(HF_ERR_ARG, "hf_k_heat_matvec: bad arguments");
    hf::k_heat_matvec_plain<<<592, 256, 0, S(stream)>>>(n, (float)h, (float)dt, (float)alpha, (float)beta, x, kap, cell_flags,
                                                       y, out);
    HF_CUDA(cudaGetLastError(), "launch (heat matvec)");
    return HF_OK;
}

}  // extern "C"
