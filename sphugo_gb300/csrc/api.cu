// api.cu -- the C ABI of include/sphgpu.h: handle lifetime, device memory
// layout, host <-> device transfers and the per-step CUDA graphs.
//
// A handle mirrors the reference's Simulation (sim/sph.go:14-21): its mutex
// plays the role of Simulation.IsBusy, it owns the particle state (kept
// resident in HBM) and counts steps. Each force evaluation is the kernel
// chain [bbox] -> bin -> scan -> permute -> knn -> density -> force,
// captured once into a CUDA graph per integration mode and replayed.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <filesystem>
#include <fstream>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

#include <cuda.h>

#include "common.cuh"

using namespace sphgpu;

namespace {
thread_local std::string g_err;

int fail(int code, const std::string &msg) {
    g_err = msg;
    return code;
}

#define CUDA_TRY(x)                                                                    \
    do {                                                                               \
        cudaError_t e_ = (x);                                                          \
        if (e_ != cudaSuccess)                                                         \
            return fail(e_ == cudaErrorMemoryAllocation ? SPH_ERR_NOMEM : SPH_ERR_CUDA, \
                        std::string(#x) + ": " + cudaGetErrorString(e_));              \
    } while (0)

// Kernel prefactors of sim/sph.go:266,275,293,303, correctly rounded (Go folds
// the constant expressions in exact arithmetic).
const double kMonahanPref = 0x1.5d3b3e3583243p+3;
const double kWendFPref = 0x1.1d34a60108f72p+1;
const double kWendDFPref = 0x1.1d34a60108f72p+2;

// Tiles shared by eight warps for lists of up to 40 entries (k <= 37), by
// four for longer lists up to k = 80; one tile per warp beyond.
int default_block_warps(int k) {
    const int need = (3 * k) / 2 + 8;
    return need <= 64 ? 8 : need <= 128 ? 4 : 0;
}

// Whether the default search is the per-query one. With few particles the
// block tiles are few (40 of 256 queries at N = 10,000, on 152 SMs), and a
// tile's chain of steps is longer than a warp per query, of which all are
// resident at once. FP64 forms, kNN stage at k = 32: N = 1000 26 us with tiles, 12
// without, 3000 33 and 14, 10,000 34 and 23, 30,000 38 and 45. At k = 16 to 64 it
// took 0.34 to 0.93 of the tiles' time, above k = 80 0.07 to 0.91 (uniform and
// clustered states, N = 400 to 16,384, ensembles of 4 x 4000 to 200 x 80), but 1.06
// at uniform N = 16,384, k = 48, and 1.4 on a perfect lattice of 16,384. The mixed form
// keeps the tiles at every size: its sums follow the order of the lists they
// leave, and a changed default would move its results in the last bits.
constexpr int64_t kPerQueryMaxN = 16384;
bool default_per_query(int64_t n, int mode) { return mode != MODE_MIXED && n <= kPerQueryMaxN; }

constexpr float kDefaultTheta = 0.5f, kDefaultHgrow = 1.04f;

int auto_level(int64_t n) {
    // about one to four particles per finest cell
    double l = std::floor(0.5 * std::log2(std::max<double>((double)n, 2.0) / 2.0) + 0.5);
    return (int)std::min<double>(std::max<double>(l, 1.0), kMaxLevel);
}
}  // namespace

void sphgpu::set_last_error(const std::string &msg) { g_err = msg; }

struct sph_handle {
    int device = 0, sms = 0;
    cudaStream_t stream = nullptr;
    int nsims = 0, k = 32, mode = MODE_EXACT64;
    int64_t n = 0;
    int64_t cap_n = 0;   // particles the per-particle arrays hold (>= n; grows on sph_append)
    int64_t n_eval = 0;  // particles whose density comes from the last force evaluation
    // frames: draw keys per caller index (empty: caller order), ranks and buffers
    std::vector<int64_t> zkeys;
    bool zrank_dirty = true;
    int32_t *d_zrank = nullptr, *d_rslot = nullptr, *d_fb = nullptr;
    uchar4 *d_rgba = nullptr;
    int64_t rank_cap = 0, fb_cap = 0;
    std::vector<sph_params> params;
    std::vector<int64_t> offs;
    std::vector<SimDev> hsims;
    SimDev *d_sims = nullptr;
    int64_t *d_offs = nullptr;
    int32_t *d_simidx = nullptr;
    unsigned *d_flags = nullptr;
    unsigned *h_flags = nullptr;  // pinned copy of the error word
    PArrays A{}, B{};
    Derived D{};
    Tables T{};
    KnnTune tune{};
    bool search_default = true;  // the search path follows k and n (not set by the caller, the tuner or a checkpoint)
    bool any_open = false, uploaded = false, evaluated = false;
    std::vector<int> base_level;  // per simulation; explicit grid_level or automatic
    std::vector<bool> auto_lvl;   // true when the level is the automatic one (the tuner may shift it)
    int level_delta = 0;
    int64_t cells_cap = 0;
    int32_t step = 0;
    cudaGraphExec_t g_step = nullptr, g_init = nullptr, g_forces = nullptr, g_prof = nullptr;
    cudaEvent_t ev[SPH_NUM_STAGES + 1] = {};
    int kernels_per_step = 0;
    double *d_io = nullptr;   // transfer / reduction staging
    size_t io_doubles = 0;
    void *d_nbr_io = nullptr; // neighbour export staging (lazy)
    std::vector<void *> allocs;
    std::vector<size_t> alloc_bytes;  // sizes of allocs, entry by entry
    std::mutex mu;

    Ctx ctx() const {
        Ctx c;
        c.sims = d_sims;
        c.sims_rw = d_sims;
        c.offs = d_offs;
        c.simidx = nsims > 1 ? d_simidx : nullptr;
        c.nsims = nsims;
        c.n = n;
        c.k = k;
        c.flags = d_flags;
        return c;
    }
    Launch launch() const { return Launch{sms, stream}; }
};

namespace sphgpu {
void para_ramp_table(unsigned char out[256 * 4]);
int set_ramp(const unsigned char rgba[256 * 4]);
void launch_render(const Ctx &c, const Launch &L, const PArrays &A, const int32_t *zrank, int32_t *rslot,
                   int32_t *fb, const double *rho, int64_t n_eval, double mass, int W, int H, uchar4 *out);
}  // namespace sphgpu

namespace {

template <typename T>
int dalloc(sph_handle *h, T **p, size_t count) {
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
    if (e != cudaSuccess) {
        *p = nullptr;
        return fail(e == cudaErrorMemoryAllocation ? SPH_ERR_NOMEM : SPH_ERR_CUDA,
                    std::string("cudaMalloc: ") + cudaGetErrorString(e));
    }
    h->allocs.push_back(q);
    h->alloc_bytes.push_back(std::max<size_t>(count, 1) * sizeof(T));
    *p = (T *)q;
    return SPH_OK;
}

void dfree(sph_handle *h, void *p) {
    if (!p) return;
    for (size_t i = 0; i < h->allocs.size(); i++)
        if (h->allocs[i] == p) {
            h->allocs.erase(h->allocs.begin() + (long)i);
            h->alloc_bytes.erase(h->alloc_bytes.begin() + (long)i);
            break;
        }
    cudaFree(p);
}

int alloc_parrays(sph_handle *h, PArrays &P, bool mixed, int64_t n) {
    int rc = 0;
    rc |= dalloc(h, &P.pos, n);
    rc |= dalloc(h, &P.vel, n);
    rc |= dalloc(h, &P.vp, n);
    rc |= dalloc(h, &P.acc, n);
    rc |= dalloc(h, &P.u, n);
    rc |= dalloc(h, &P.up, n);
    rc |= dalloc(h, &P.udot, n);
    rc |= dalloc(h, &P.id, n);
    rc |= dalloc(h, &P.hprev, n);
    rc |= dalloc(h, &P.rec, n);
    if (mixed) rc |= dalloc(h, &P.vrec, n);  // predicted velocities as float pairs
    return rc ? SPH_ERR_NOMEM : SPH_OK;
}

// Every per-particle array (state, evaluation copy, derived values, binning
// keys, staging) for `cap` particles.
int alloc_particles(sph_handle *h, int64_t cap) {
    const bool mixed = h->mode == MODE_MIXED;
    const int64_t k = h->k;
    int rc = alloc_parrays(h, h->A, mixed, cap) | alloc_parrays(h, h->B, mixed, cap);
    rc |= dalloc(h, &h->D.rho, cap);
    rc |= dalloc(h, &h->D.c, cap);
    rc |= dalloc(h, &h->D.h, cap);
    rc |= dalloc(h, &h->D.nbr, cap * k);
    rc |= dalloc(h, &h->D.defer, cap);
    if (mixed) {
        rc |= dalloc(h, &h->D.derf, cap);
        rc |= dalloc(h, &h->D.d2f, cap * k);
    } else {
        rc |= dalloc(h, &h->D.der, cap);
        rc |= dalloc(h, &h->D.dist, cap * k);
    }
    rc |= dalloc(h, &h->T.key, cap);
    rc |= dalloc(h, &h->T.rank, cap);
    rc |= dalloc(h, &h->T.tmp, cap);
    h->io_doubles = (size_t)std::max<int64_t>(8 * cap, 3 * cap + 512);
    rc |= dalloc(h, &h->d_io, h->io_doubles);
    h->cap_n = cap;
    return rc ? SPH_ERR_NOMEM : SPH_OK;
}

// Draw keys of appended particles (sph_append): kept only once keys exist.
void draw_keys_append(sph_handle *h, int64_t n0, int64_t count, const int64_t *z) {
    if (!z && h->zkeys.empty()) return;
    if (h->zkeys.empty())
        for (int64_t i = 0; i < n0; i++) h->zkeys.push_back(-i);  // caller order
    for (int64_t i = 0; i < count; i++) h->zkeys.push_back(z ? z[i] : -(n0 + i));
    h->zrank_dirty = true;
}

int check_params(const sph_params &p, int64_t n) {
    if (p.k < 1 || p.k > 128) return fail(SPH_ERR_ARG, "k must be in [1, 128]");
    if (n < (int64_t)p.k + 1) return fail(SPH_ERR_ARG, "a simulation needs at least k+1 particles");
    if (p.kernel != SPH_KERNEL_MONAHAN && p.kernel != SPH_KERNEL_WENDLAND)
        return fail(SPH_ERR_ARG, "unknown kernel");
    if (p.precision < 0 || p.precision > 2) return fail(SPH_ERR_ARG, "unknown precision");
    if (p.grid_level < 0 || p.grid_level > kMaxLevel) return fail(SPH_ERR_ARG, "grid_level must be in [0, 14]");
    const double *ax[2] = {p.hor, p.vert};
    for (int a = 0; a < 2; a++) {
        // sim/nearest-neighbour.go:39-55 panics on a half-open axis
        if (ax[a][0] == -DBL_MAX) {
            if (ax[a][1] != DBL_MAX) return fail(SPH_ERR_ARG, "cannot have open and periodic boundary on one axis");
        } else if (!(ax[a][1] > ax[a][0]) || !std::isfinite(ax[a][1] - ax[a][0])) {
            return fail(SPH_ERR_ARG, "periodic bounds must satisfy lo < hi");
        }
    }
    if (!std::isfinite(p.dth) || !std::isfinite(p.gamma) || !std::isfinite(p.mass))
        return fail(SPH_ERR_ARG, "non-finite parameter");
    return SPH_OK;
}

SimDev make_simdev(const sph_params &p, int64_t off, int64_t n, int64_t cell_off, int level) {
    SimDev S;
    memset(&S, 0, sizeof S);
    S.off = off;
    S.n = n;
    S.cell_off = cell_off;
    S.level = level;
    S.kernel = p.kernel;
    const double *ax[2] = {p.hor, p.vert};
    int G = 1 << level;
    for (int a = 0; a < 2; a++) {
        S.per_lo[a] = ax[a][0];
        S.per_hi[a] = ax[a][1];
        S.periodic[a] = ax[a][0] != -DBL_MAX;
        if (S.periodic[a]) {
            S.lo[a] = ax[a][0];
            S.L[a] = ax[a][1] - ax[a][0];
            S.dimg[a] = ax[a][1] - ax[a][0];
        } else {
            S.lo[a] = 0.0;
            S.L[a] = 1.0;
            S.dimg[a] = 0.0;
        }
        S.s[a] = S.L[a] / G;
        S.inv_s[a] = G / S.L[a];
    }
    S.gamma = p.gamma;
    S.mass = p.mass;
    S.dth = p.dth;
    S.accel[0] = p.accel[0];
    S.accel[1] = p.accel[1];
    // a NaN bound reflects nothing, as an infinite one (the force compares bounds as integers)
    for (int i = 0; i < 4; i++) S.refl[i] = std::isnan(p.refl[i]) ? (i & 1 ? HUGE_VAL : -HUGE_VAL) : p.refl[i];
    S.alpha = p.alpha;
    S.beta = p.beta;
    S.etasq = p.etasq;
    S.fpref = p.kernel == SPH_KERNEL_WENDLAND ? kWendFPref : kMonahanPref;
    S.dfpref = p.kernel == SPH_KERNEL_WENDLAND ? kWendDFPref : kMonahanPref;
    reset_reductions(S);
    S.tol = (float)(std::max(S.L[0], S.L[1]) * 4.0e-7);
    simdev_floats(S);
    simdev_fcell(S);
    return S;
}

void destroy_graphs(sph_handle *h) {
    if (h->g_step) cudaGraphExecDestroy(h->g_step);
    if (h->g_init) cudaGraphExecDestroy(h->g_init);
    if (h->g_forces) cudaGraphExecDestroy(h->g_forces);
    if (h->g_prof) cudaGraphExecDestroy(h->g_prof);
    h->g_step = h->g_init = h->g_forces = h->g_prof = nullptr;
}

// One force evaluation (plus the integration when `integrate`); with
// `events`, an event is recorded before each stage and after the last.
void enqueue_eval(sph_handle *h, int pred, bool integrate, bool events = false) {
    Ctx c = h->ctx();
    Launch L = h->launch();
    auto mark = [&](int i) {
        // external event nodes (plain records only order work inside a capture)
        if (events) cudaEventRecordWithFlags(h->ev[i], h->stream, cudaEventRecordExternal);
    };
    mark(0);
    if (h->any_open) launch_bbox(c, L, h->A, pred);
    launch_bin(c, L, h->A, h->T, h->D.ndefer, pred);
    mark(1);
    launch_scan(c, L, h->T);
    mark(2);
    launch_permute(c, L, h->A, h->B, h->T, pred, h->mode == MODE_MIXED);  // velocity records: the mixed force reads them
    mark(3);
    const int mode = kernel_mode(h->mode);
    launch_knn(c, L, h->B, h->D, h->T, mode, h->tune);
    mark(4);
    launch_density(c, L, h->B, h->D, mode, &h->tune);
    mark(5);
    launch_force(c, L, h->B, h->A, h->D, mode, integrate);
    mark(6);
}

int count_kernel_nodes(cudaGraph_t g) {
    size_t n = 0;
    if (cudaGraphGetNodes(g, nullptr, &n) != cudaSuccess) return 0;
    std::vector<cudaGraphNode_t> nodes(n);
    cudaGraphGetNodes(g, nodes.data(), &n);
    int k = 0;
    for (auto nd : nodes) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) k++;
    }
    return k;
}

int capture(sph_handle *h, int pred, bool integrate, cudaGraphExec_t *out, bool events = false,
            int *kernels = nullptr) {
    cudaGraph_t g = nullptr;
    CUDA_TRY(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    enqueue_eval(h, pred, integrate, events);
    CUDA_TRY(cudaStreamEndCapture(h->stream, &g));
    if (kernels) *kernels = count_kernel_nodes(g);
    cudaError_t e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(SPH_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    return SPH_OK;
}

int check_flags(sph_handle *h) {
    CUDA_TRY(cudaMemcpyAsync(h->h_flags, h->d_flags, sizeof(unsigned), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    const unsigned f = *h->h_flags;
    if (!f) return SPH_OK;
    CUDA_TRY(cudaMemsetAsync(h->d_flags, 0, sizeof(unsigned), h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    if (f & FLAG_SENTINEL)
        return fail(SPH_ERR_SENTINEL, "a k-th neighbour lies at squared distance >= 0.4, beyond the reference's queue sentinel");
    if (f & FLAG_KNN_FEW) return fail(SPH_ERR_KNN, "fewer than k neighbour candidates exist for some particle");
    if (f & FLAG_KNN_ATTEMPTS) return fail(SPH_ERR_KNN, "neighbour search radius did not converge");
    if (f & FLAG_NONFINITE) return fail(SPH_ERR_RANGE, "non-finite particle position");
    return fail(SPH_ERR_RANGE, "kernel argument q outside [0,1] or non-finite force");
}

int ensure_graphs(sph_handle *h) {
    int rc;
    if (!h->g_step && (rc = capture(h, PRED_DRIFT, true, &h->g_step, false, &h->kernels_per_step))) return rc;
    if (!h->g_init && (rc = capture(h, PRED_INIT, false, &h->g_init))) return rc;
    if (!h->g_forces && (rc = capture(h, PRED_KEEP, false, &h->g_forces))) return rc;
    return SPH_OK;
}

struct Guard {
    sph_handle *h;
    std::lock_guard<std::mutex> lk;
    explicit Guard(sph_handle *hh) : h(hh), lk(hh->mu) { cudaSetDevice(hh->device); }
};

int create_impl(const sph_params *params, const int64_t *counts, int32_t nsims, sph_handle **out) {
    if (!out) return fail(SPH_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (!params || !counts || nsims < 1) return fail(SPH_ERR_ARG, "need at least one simulation");
    int64_t total = 0;
    for (int s = 0; s < nsims; s++) {
        int rc = check_params(params[s], counts[s]);
        if (rc) return rc;
        if (params[s].k != params[0].k || params[s].precision != params[0].precision)
            return fail(SPH_ERR_ARG, "k and precision must agree across an ensemble");
        total += counts[s];
    }
    if (total >= kMaxParticles) return fail(SPH_ERR_ARG, "too many particles (limit 2^27)");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
        cudaGetLastError();
        return fail(SPH_ERR_CUDA, "no CUDA device available");
    }
    sph_handle *h = new sph_handle();
    cudaGetDevice(&h->device);
    cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device);
    h->nsims = nsims;
    h->n = total;
    h->k = params[0].k;
    h->mode = params[0].precision == SPH_PREC_MIXED       ? MODE_MIXED
              : params[0].precision == SPH_PREC_FP64_FAST ? MODE_FAST64
                                                          : MODE_EXACT64;
    h->params.assign(params, params + nsims);
    h->offs.resize(nsims + 1);
    h->offs[0] = 0;
    int64_t cells = 0, cap = 0;
    for (int s = 0; s < nsims; s++) {
        h->offs[s + 1] = h->offs[s] + counts[s];
        const bool autol = params[s].grid_level <= 0;
        int level = autol ? auto_level(counts[s]) : params[s].grid_level;
        h->base_level.push_back(level);
        h->auto_lvl.push_back(autol);
        h->hsims.push_back(make_simdev(params[s], h->offs[s], counts[s], cells, level));
        h->any_open = h->any_open || !h->hsims.back().periodic[0] || !h->hsims.back().periodic[1];
        cells += (int64_t)1 << (2 * level);
        // room for the tuner to refine an automatic level by up to two
        cap += (int64_t)1 << (2 * (autol ? std::min(level + 2, kMaxLevel) : level));
    }
    h->cells_cap = cap;
    if (cap >= ((int64_t)1 << 31) - 1) {
        delete h;
        return fail(SPH_ERR_ARG, "cell tables exceed 2^31 cells; lower grid_level");
    }
    int rc = 0;
    auto bail = [&](int code) {
        std::string m = g_err;
        sph_destroy(h);
        g_err = m;
        return code;
    };
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(fail(SPH_ERR_CUDA, "cudaStreamCreate failed"));
    const int64_t n = h->n, k = h->k;
    if (cudaHostAlloc((void **)&h->h_flags, sizeof(unsigned), cudaHostAllocDefault) != cudaSuccess)
        return bail(fail(SPH_ERR_NOMEM, "cudaHostAlloc failed"));
    rc |= dalloc(h, &h->d_sims, nsims);
    rc |= dalloc(h, &h->d_offs, nsims + 1);
    if (nsims > 1) rc |= dalloc(h, &h->d_simidx, total);
    rc |= dalloc(h, &h->d_flags, 2);
    if (rc) return bail(SPH_ERR_NOMEM);
    if (alloc_particles(h, n)) return bail(SPH_ERR_NOMEM);
    rc |= dalloc(h, &h->D.ndefer, 2);
    h->T.ncells = cells;
    rc |= dalloc(h, &h->T.count, cap);
    rc |= dalloc(h, &h->T.start, cap + 1);
    rc |= dalloc(h, &h->T.partial, cap / 4096 + 2);
    if (rc) return bail(SPH_ERR_NOMEM);
    if (cudaMemset(h->T.count, 0, cap * sizeof(int32_t)) != cudaSuccess ||
        cudaMemset(h->D.nbr, 0, n * k * sizeof(int32_t)) != cudaSuccess ||
        cudaMemset(h->B.id, 0, n * sizeof(int32_t)) != cudaSuccess ||
        cudaMemset(h->A.id, 0, n * sizeof(int32_t)) != cudaSuccess ||
        cudaMemset(h->d_flags, 0, 2 * sizeof(unsigned)) != cudaSuccess ||
        cudaMemset(h->A.hprev, 0, n * sizeof(float)) != cudaSuccess ||
        cudaMemcpy(h->d_sims, h->hsims.data(), nsims * sizeof(SimDev), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->d_offs, h->offs.data(), (nsims + 1) * sizeof(int64_t), cudaMemcpyHostToDevice) != cudaSuccess)
        return bail(fail(SPH_ERR_CUDA, "device initialisation failed"));
    if (nsims > 1) {
        std::vector<int32_t> idx((size_t)total);
        for (int s = 0; s < nsims; s++)
            for (int64_t i = h->offs[s]; i < h->offs[s + 1]; i++) idx[(size_t)i] = s;
        if (cudaMemcpy(h->d_simidx, idx.data(), total * sizeof(int32_t), cudaMemcpyHostToDevice) != cudaSuccess)
            return bail(fail(SPH_ERR_CUDA, "device initialisation failed"));
    }
    knn_init_attrs();
    h->tune.block = 256;
    h->tune.cap = (int)(k + 16);
    h->tune.theta = kDefaultTheta;
    h->tune.hgrow = kDefaultHgrow;
    h->tune.blocks_per_sm = std::max(1, knn_occupancy_blocks(h->tune.block, h->tune.cap, kernel_mode(h->mode)));
    h->tune.tile = default_per_query(n, h->mode) ? 0 : 1;
    h->tune.tile_blocks_per_sm = std::max(1, knn_tile_occupancy_blocks((int)k, kernel_mode(h->mode)));
    h->tune.block_warps = default_block_warps((int)k);
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return bail(fail(SPH_ERR_CUDA, cudaGetErrorString(e)));
    *out = h;
    return SPH_OK;
}

// The device's address of `bytes` bytes of the caller's memory when all of
// them are pinned and mapped (cudaHostAlloc, cudaHostRegister), else NULL. The
// kernels then read and write them in place: one pass over the host link
// instead of a copy into a staging array and a pass over that (set_state,
// get_state and get_derived of N = 4,194,304: 1.81, 2.26 and 0.70 ms with the
// copies, 1.33, 1.44 and 0.57 in place, 202, 186 and 178 GB/s), and with few
// particles two kernels instead of eight copies (N = 10,000: 41, 36 and 22 us,
// 25, 25 and 18 in place).
void *mapped_host(const void *p, size_t bytes) {
    typedef CUresult (*GetAttributes)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
    static const GetAttributes get = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (GetAttributes)f;
    }();
    if (!get || !p || !bytes) return nullptr;
    unsigned type = 0, managed = 0, access = 0;
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute which[6] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                    CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                    CU_POINTER_ATTRIBUTE_RANGE_SIZE, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
    void *out[6] = {&type, &managed, &dev, &start, &size, &access};
    if (get(6, which, out, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS) return nullptr;
    // (the range may be given by the host's or the device's address)
    const uintptr_t off = (uintptr_t)start <= (uintptr_t)p && (uintptr_t)p - (uintptr_t)start < size
                              ? (uintptr_t)p - (uintptr_t)start
                              : (uintptr_t)dev - (uintptr_t)start;
    if (type != CU_MEMORYTYPE_HOST || managed || access != 3u /* read and write */ || !dev || off > size || bytes > size - off) return nullptr;
    if ((uintptr_t)dev % alignof(double)) return nullptr;
    return (void *)(uintptr_t)dev;
}

// Where a kernel finds the caller's n values: in place, or in the staging
// array after a copy.
int stage_in(sph_handle *h, double *staging, const double *src, const double **dev) {
    *dev = nullptr;
    if (!src) return SPH_OK;
    if (void *m = mapped_host(src, h->n * sizeof(double))) {
        *dev = (const double *)m;
        return SPH_OK;
    }
    CUDA_TRY(cudaMemcpyAsync(staging, src, h->n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    *dev = staging;
    return SPH_OK;
}
// The map (in the binning's scratch) to the caller's order for a transfer with an
// array in place; a transfer through staging arrays alone runs in the slots' order,
// without one, unless it reads more than kSlotOrderMaxN particles out: its scattered
// writes then cost more than scattered reads once the arrays outgrow L2. Pageable
// host arrays, us, caller's order and the slots': set_state N = 10,000 108 and 103,
// 1,048,576 570 and 535, 4,194,304 2668 and 2168; get_state 10,000 106 and 98,
// 1,048,576 496 and 492, 2,097,152 933 and 1156, 4,194,304 1870 and 2578; get_derived
// 51 and 41, 195 and 187, 350 and 335, 699 and 728.
constexpr int64_t kSlotOrderMaxN = (int64_t)1 << 20;
template <typename T>
const int32_t *slots_for(sph_handle *h, T *const *dev, int arrays, bool out) {
    bool map = out && h->n > kSlotOrderMaxN;
    for (int i = 0; i < arrays; i++) map |= dev[i] && (dev[i] < h->d_io || dev[i] >= h->d_io + h->io_doubles);
    if (!map) return nullptr;
    launch_slots(h->ctx(), h->launch(), h->A, h->T.tmp);
    return h->T.tmp;
}
// Where a kernel leaves n values for the caller: in place, or in the staging
// array, which copy_out then brings over.
double *stage_out(sph_handle *h, double *staging, double *dst) {
    if (!dst) return nullptr;
    void *m = mapped_host(dst, h->n * sizeof(double));
    return m ? (double *)m : staging;
}
int copy_out(sph_handle *h, double *dst, const double *src, const double *staging) {
    if (!dst || src != staging) return SPH_OK;
    CUDA_TRY(cudaMemcpyAsync(dst, src, h->n * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    return SPH_OK;
}

// ------------------------------------------------------------------ tuning
// Rebuilds the cell-table layout for binning levels base + delta (automatic
// levels only); graphs captured with the old layout are dropped.
int apply_levels(sph_handle *h, int delta) {
    int64_t cells = 0;
    for (int s = 0; s < h->nsims; s++) {
        int level = h->base_level[s];
        if (h->auto_lvl[s]) level = std::min(std::max(level + delta, 1), kMaxLevel);
        SimDev S = make_simdev(h->params[s], h->offs[s], h->offs[s + 1] - h->offs[s], cells, level);
        h->hsims[s] = S;
        cells += (int64_t)1 << (2 * level);
    }
    if (cells > h->cells_cap) return fail(SPH_ERR_ARG, "binning level beyond the allocated cell table");
    CUDA_TRY(cudaMemcpyAsync(h->d_sims, h->hsims.data(), h->nsims * sizeof(SimDev), cudaMemcpyHostToDevice,
                             h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    h->T.ncells = cells;
    h->level_delta = delta;
    destroy_graphs(h);
    return SPH_OK;
}

// Mean device time of one forces-only evaluation (after one untimed one that
// lets the radius guess settle on the previous smoothing lengths).
int time_forces(sph_handle *h, int reps, double *ms) {
    int rc = ensure_graphs(h);
    if (rc) return rc;
    if (!h->ev[0])
        for (auto &e : h->ev) CUDA_TRY(cudaEventCreate(&e));
    CUDA_TRY(cudaGraphLaunch(h->g_forces, h->stream));
    CUDA_TRY(cudaEventRecord(h->ev[0], h->stream));
    for (int r = 0; r < reps; r++) CUDA_TRY(cudaGraphLaunch(h->g_forces, h->stream));
    CUDA_TRY(cudaEventRecord(h->ev[1], h->stream));
    CUDA_TRY(cudaEventSynchronize(h->ev[1]));
    float t = 0.f;
    CUDA_TRY(cudaEventElapsedTime(&t, h->ev[0], h->ev[1]));
    *ms = t / reps;
    return check_flags(h);
}

std::string tune_cache_path() {
    if (const char *p = std::getenv("SPHGPU_TUNE_CACHE")) return p;
    const char *home = std::getenv("HOME");
    return std::string(home ? home : "/tmp") + "/.cache/sphgpu/tune.txt";
}

struct TuneChoice {
    float theta = kDefaultTheta, hgrow = kDefaultHgrow;
    int delta = 0, tile = 1, block = 8;
    double ms = 0.0;
};

std::string tune_key(const sph_handle *h, const char *dist) {
    std::ostringstream o;
    const int nb = (int)std::lround(2.0 * std::log2((double)std::max<int64_t>(h->n, 1)));
    o << "nb=" << nb << " k=" << h->k << " form=" << h->mode << " sims=" << (h->nsims > 1 ? 2 : 1)
      << " dist=" << dist;
    return o.str();
}

bool tune_cache_get(const std::string &key, TuneChoice *c) {
    std::ifstream f(tune_cache_path());
    std::string line;
    bool found = false;
    while (std::getline(f, line)) {
        if (line.rfind("sphgpu-tune-v3 " + key + " ", 0) != 0) continue;
        std::istringstream in(line.substr(16 + key.size()));
        std::string tok;
        while (in >> tok) {
            const size_t eq = tok.find('=');
            if (eq == std::string::npos) continue;
            const std::string k = tok.substr(0, eq), v = tok.substr(eq + 1);
            if (k == "theta") c->theta = std::stof(v);
            else if (k == "hgrow") c->hgrow = std::stof(v);
            else if (k == "delta") c->delta = std::stoi(v);
            else if (k == "tile") c->tile = std::stoi(v);
            else if (k == "block") c->block = std::stoi(v);
            else if (k == "ms") c->ms = std::stod(v);
        }
        found = true;  // the last matching line wins
    }
    return found;
}

void tune_cache_put(const std::string &key, const TuneChoice &c) {
    const std::string path = tune_cache_path();
    std::error_code ec;
    std::filesystem::create_directories(std::filesystem::path(path).parent_path(), ec);
    std::ofstream f(path, std::ios::app);
    if (!f) return;
    f << "sphgpu-tune-v3 " << key << " theta=" << c.theta << " hgrow=" << c.hgrow << " delta=" << c.delta
      << " tile=" << c.tile << " block=" << c.block << " ms=" << c.ms << "\n";
}

}  // namespace

// ======================================================================= ABI
extern "C" {

sph_params sph_default_params(void) {
    sph_params p;
    memset(&p, 0, sizeof p);
    p.k = 32;
    p.kernel = SPH_KERNEL_MONAHAN;
    p.precision = SPH_PREC_FP64;
    p.grid_level = 0;
    p.gamma = 1.66666;
    p.mass = 1.0;
    p.dth = 0.001;
    p.hor[0] = -DBL_MAX;
    p.hor[1] = DBL_MAX;
    p.vert[0] = -DBL_MAX;
    p.vert[1] = DBL_MAX;
    p.refl[0] = -DBL_MAX;
    p.refl[1] = DBL_MAX;
    p.refl[2] = -DBL_MAX;
    p.refl[3] = DBL_MAX;
    p.alpha = 0.75;
    p.beta = 1.5;
    p.etasq = 0.01;
    return p;
}

int32_t sph_abi_version(void) { return SPHGPU_ABI_VERSION; }

const char *sph_last_error(void) { return g_err.c_str(); }

int sph_device_count(int32_t *count) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (count) *count = 0;
        return fail(SPH_ERR_CUDA, cudaGetErrorString(e));
    }
    if (count) *count = n;
    return SPH_OK;
}

int sph_create(const sph_params *p, int64_t n, sph_handle **out) { return create_impl(p, &n, 1, out); }

int sph_ens_create(const sph_params *params, const int64_t *counts, int32_t nsims, sph_handle **out) {
    return create_impl(params, counts, nsims, out);
}

int sph_destroy(sph_handle *h) {
    if (!h) return SPH_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    destroy_graphs(h);
    for (void *p : h->allocs) cudaFree(p);
    if (h->d_nbr_io) cudaFree(h->d_nbr_io);
    if (h->h_flags) cudaFreeHost(h->h_flags);
    for (auto &e : h->ev)
        if (e) cudaEventDestroy(e);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return SPH_OK;
}

int sph_upload(sph_handle *h, const double *x, const double *y, const double *vx, const double *vy,
               const double *u) {
    if (!h || !x || !y) return fail(SPH_ERR_ARG, "handle, x and y are required");
    Guard g(h);
    const int64_t n = h->n;
    const double *src[5] = {x, y, vx, vy, u}, *d[5];
    for (int i = 0; i < 5; i++)
        if (int rc = stage_in(h, h->d_io + i * n, src[i], &d[i])) return rc;
    launch_scatter_state(h->ctx(), h->launch(), h->A, nullptr, d[0], d[1], d[2], d[3], d[4], nullptr, nullptr, nullptr, true);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    h->step = 0;
    h->uploaded = true;
    h->evaluated = false;
    return SPH_OK;
}

int sph_append(sph_handle *h, int64_t count, const double *x, const double *y, const double *vx,
               const double *vy, const double *u, const int64_t *z) {
    if (!h || count < 0 || (count > 0 && (!x || !y))) return fail(SPH_ERR_ARG, "bad handle, count or arrays");
    Guard g(h);
    if (h->nsims != 1) return fail(SPH_ERR_ARG, "particles can be appended to a single simulation only");
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_append before sph_upload");
    if (count == 0) return SPH_OK;
    const int64_t n0 = h->n, n1 = n0 + count;
    if (n1 >= kMaxParticles) return fail(SPH_ERR_ARG, "too many particles (limit 2^27)");
    if (n1 > h->cap_n) {
        // grow like a Go slice; only the state needs copying (the rest is rebuilt per evaluation)
        const int64_t cap = std::min<int64_t>(std::max<int64_t>(n1, h->cap_n + h->cap_n / 2), kMaxParticles);
        const PArrays oldA = h->A, oldB = h->B;
        const Derived oldD = h->D;
        const Tables oldT = h->T;
        double *old_io = h->d_io;
        const int64_t old_cap = h->cap_n;
        const size_t old_io_doubles = h->io_doubles;
        if (alloc_particles(h, cap)) {
            // release whatever the failed attempt got and keep the old arrays
            const PArrays newA = h->A, newB = h->B;
            const Derived newD = h->D;
            const Tables newT = h->T;
            double *new_io = h->d_io;
            auto drop = [&](void *nw, void *old) {
                if (nw && nw != old) dfree(h, nw);
            };
            drop(newA.pos, oldA.pos); drop(newA.vel, oldA.vel); drop(newA.vp, oldA.vp); drop(newA.acc, oldA.acc);
            drop(newA.u, oldA.u); drop(newA.up, oldA.up); drop(newA.udot, oldA.udot); drop(newA.id, oldA.id);
            drop(newA.hprev, oldA.hprev); drop(newA.rec, oldA.rec); drop(newA.vrec, oldA.vrec);
            drop(newB.pos, oldB.pos); drop(newB.vel, oldB.vel); drop(newB.vp, oldB.vp); drop(newB.acc, oldB.acc);
            drop(newB.u, oldB.u); drop(newB.up, oldB.up); drop(newB.udot, oldB.udot); drop(newB.id, oldB.id);
            drop(newB.hprev, oldB.hprev); drop(newB.rec, oldB.rec); drop(newB.vrec, oldB.vrec);
            drop(newD.rho, oldD.rho); drop(newD.c, oldD.c); drop(newD.h, oldD.h); drop(newD.nbr, oldD.nbr);
            drop(newD.defer, oldD.defer); drop(newD.der, oldD.der); drop(newD.derf, oldD.derf);
            drop(newD.dist, oldD.dist); drop(newD.d2f, oldD.d2f);
            drop(newT.key, oldT.key); drop(newT.rank, oldT.rank); drop(newT.tmp, oldT.tmp);
            drop(new_io, old_io);
            h->A = oldA;
            h->B = oldB;
            h->D = oldD;
            h->T = oldT;
            h->d_io = old_io;
            h->cap_n = old_cap;
            h->io_doubles = old_io_doubles;
            return fail(SPH_ERR_NOMEM, "cannot grow the particle arrays");
        }
        h->D.ndefer = oldD.ndefer;
        h->T.count = oldT.count;
        h->T.start = oldT.start;
        h->T.partial = oldT.partial;
        h->T.ncells = oldT.ncells;
        auto cp = [&](void *dst, const void *src, size_t bytes) {
            return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, h->stream);
        };
        CUDA_TRY(cp(h->A.pos, oldA.pos, n0 * sizeof(double2)));
        CUDA_TRY(cp(h->A.vel, oldA.vel, n0 * sizeof(double2)));
        CUDA_TRY(cp(h->A.vp, oldA.vp, n0 * sizeof(double2)));
        CUDA_TRY(cp(h->A.acc, oldA.acc, n0 * sizeof(double2)));
        CUDA_TRY(cp(h->A.u, oldA.u, n0 * sizeof(double)));
        CUDA_TRY(cp(h->A.up, oldA.up, n0 * sizeof(double)));
        CUDA_TRY(cp(h->A.udot, oldA.udot, n0 * sizeof(double)));
        CUDA_TRY(cp(h->A.id, oldA.id, n0 * sizeof(int32_t)));
        CUDA_TRY(cp(h->A.hprev, oldA.hprev, n0 * sizeof(float)));
        CUDA_TRY(cp(h->D.rho, oldD.rho, n0 * sizeof(double)));  // densities of the last evaluation (frames)
        CUDA_TRY(cudaMemsetAsync(h->D.nbr, 0, (size_t)cap * h->k * sizeof(int32_t), h->stream));
        CUDA_TRY(cudaStreamSynchronize(h->stream));
        for (const PArrays *P : {&oldA, &oldB})
            for (void *q : {(void *)P->pos, (void *)P->vel, (void *)P->vp, (void *)P->acc, (void *)P->u,
                            (void *)P->up, (void *)P->udot, (void *)P->id, (void *)P->hprev, (void *)P->rec,
                            (void *)P->vrec})
                dfree(h, q);
        for (void *q : {(void *)oldD.rho, (void *)oldD.c, (void *)oldD.h, (void *)oldD.nbr, (void *)oldD.defer,
                        (void *)oldD.der, (void *)oldD.derf, (void *)oldD.dist, (void *)oldD.d2f,
                        (void *)oldT.key, (void *)oldT.rank, (void *)oldT.tmp, (void *)old_io})
            dfree(h, q);
        if (h->d_nbr_io) {
            cudaFree(h->d_nbr_io);
            h->d_nbr_io = nullptr;
        }
    }
    double *d = h->d_io;
    const double *src[5] = {x, y, vx, vy, u};
    for (int a = 0; a < 5; a++) {
        if (src[a]) CUDA_TRY(cudaMemcpyAsync(d + a * count, src[a], count * sizeof(double), cudaMemcpyHostToDevice, h->stream));
        else CUDA_TRY(cudaMemsetAsync(d + a * count, 0, count * sizeof(double), h->stream));
    }
    launch_append(h->launch(), h->A, n0, count, d);
    CUDA_TRY(cudaGetLastError());
    h->n = n1;
    h->offs[1] = n1;
    h->hsims[0].n = n1;
    CUDA_TRY(cudaMemcpyAsync(h->d_sims, h->hsims.data(), sizeof(SimDev), cudaMemcpyHostToDevice, h->stream));
    CUDA_TRY(cudaMemcpyAsync(h->d_offs, h->offs.data(), 2 * sizeof(int64_t), cudaMemcpyHostToDevice, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    draw_keys_append(h, n0, count, z);
    if (h->search_default) h->tune.tile = default_per_query(n1, h->mode) ? 0 : 1;
    destroy_graphs(h);
    return SPH_OK;
}

int sph_set_state(sph_handle *h, const double *x, const double *y, const double *vx, const double *vy,
                  const double *u, const double *ax, const double *ay, const double *udot) {
    if (!h || !x || !y) return fail(SPH_ERR_ARG, "handle, x and y are required");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_set_state before sph_upload");
    const int64_t n = h->n;
    const double *src[8] = {x, y, vx, vy, u, ax, ay, udot}, *d[8];
    for (int i = 0; i < 8; i++)
        if (int rc = stage_in(h, h->d_io + i * n, src[i], &d[i])) return rc;
    launch_scatter_state(h->ctx(), h->launch(), h->A, slots_for(h, d, 8, false), d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], false);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

int sph_get_state(sph_handle *h, double *x, double *y, double *vx, double *vy, double *u, double *ax,
                  double *ay, double *udot) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "no state uploaded");
    const int64_t n = h->n;
    double *dst[8] = {x, y, vx, vy, u, ax, ay, udot}, *d[8];
    for (int i = 0; i < 8; i++) d[i] = stage_out(h, h->d_io + i * n, dst[i]);
    launch_gather_state(h->ctx(), h->launch(), h->A, slots_for(h, d, 8, true), d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7]);
    CUDA_TRY(cudaGetLastError());
    for (int i = 0; i < 8; i++)
        if (int rc = copy_out(h, dst[i], d[i], h->d_io + i * n)) return rc;
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

int sph_get_derived(sph_handle *h, double *rho, double *c, double *hsml) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "no state uploaded");
    const int64_t n = h->n;
    double *dst[3] = {rho, c, hsml}, *d[3];
    for (int i = 0; i < 3; i++) d[i] = stage_out(h, h->d_io + i * n, dst[i]);
    launch_gather_derived(h->ctx(), h->launch(), h->A, h->D, slots_for(h, d, 3, true), d[0], d[1], d[2]);
    CUDA_TRY(cudaGetLastError());
    for (int i = 0; i < 3; i++)
        if (int rc = copy_out(h, dst[i], d[i], h->d_io + i * n)) return rc;
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

int sph_memory_bytes(sph_handle *h, int64_t *bytes) {
    if (!h || !bytes) return fail(SPH_ERR_ARG, "bad argument");
    Guard g(h);
    size_t t = 0;
    for (size_t b : h->alloc_bytes) t += b;
    *bytes = (int64_t)t;
    return SPH_OK;
}

int sph_error_norms(sph_handle *h, double *anorm, double *unorm) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (h->mode != MODE_EXACT64) return fail(SPH_ERR_STATE, "sph_error_norms needs an SPH_PREC_FP64 handle");
    if (!h->uploaded || !h->evaluated || h->n_eval != h->n) return fail(SPH_ERR_STATE, "no force evaluation yet");
    const int64_t n = h->n;
    double *d = h->d_io;
    launch_error_norms(h->ctx(), h->launch(), h->B, h->D, d, d + n);
    CUDA_TRY(cudaGetLastError());
    int rc;
    if ((rc = copy_out(h, anorm, d, d)) || (rc = copy_out(h, unorm, d + n, d + n))) return rc;
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

int sph_get_neighbours(sph_handle *h, int64_t *ids, double *dist, int32_t *img) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (!h->uploaded || !h->evaluated) return fail(SPH_ERR_STATE, "no force evaluation yet");
    const int64_t nk = h->n * h->k;
    if (!h->d_nbr_io) CUDA_TRY(cudaMalloc(&h->d_nbr_io, nk * (8 + 8 + 4)));
    int64_t *di = (int64_t *)h->d_nbr_io;
    double *dd = (double *)(di + nk);
    int32_t *dm = (int32_t *)(dd + nk);
    launch_gather_neighbours(h->ctx(), h->launch(), h->B, h->D, ids ? di : nullptr, dist ? dd : nullptr,
                             img ? dm : nullptr);
    CUDA_TRY(cudaGetLastError());
    if (ids) CUDA_TRY(cudaMemcpyAsync(ids, di, nk * 8, cudaMemcpyDeviceToHost, h->stream));
    if (dist) CUDA_TRY(cudaMemcpyAsync(dist, dd, nk * 8, cudaMemcpyDeviceToHost, h->stream));
    if (img) CUDA_TRY(cudaMemcpyAsync(img, dm, nk * 4, cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

int sph_step(sph_handle *h, int32_t nsteps) {
    if (!h || nsteps < 0) return fail(SPH_ERR_ARG, "bad handle or step count");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_step before sph_upload");
    int rc = ensure_graphs(h);
    if (rc) return rc;
    for (int32_t s = 0; s < nsteps; s++) {
        if (h->step == 0) CUDA_TRY(cudaGraphLaunch(h->g_init, h->stream));
        CUDA_TRY(cudaGraphLaunch(h->g_step, h->stream));
        h->step++;
    }
    if (nsteps > 0) {
        h->evaluated = true;
        h->n_eval = h->n;
    }
    return check_flags(h);
}

int sph_forces(sph_handle *h) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_forces before sph_upload");
    int rc = ensure_graphs(h);
    if (rc) return rc;
    CUDA_TRY(cudaGraphLaunch(h->g_forces, h->stream));
    h->evaluated = true;
    h->n_eval = h->n;
    return check_flags(h);
}

int sph_step_async(sph_handle *h, int32_t nsteps) {
    if (!h || nsteps < 0) return fail(SPH_ERR_ARG, "bad handle or step count");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_step_async before sph_upload");
    int rc = ensure_graphs(h);
    if (rc) return rc;
    for (int32_t s = 0; s < nsteps; s++) {
        if (h->step == 0) CUDA_TRY(cudaGraphLaunch(h->g_init, h->stream));
        CUDA_TRY(cudaGraphLaunch(h->g_step, h->stream));
        h->step++;
    }
    if (nsteps > 0) {
        h->evaluated = true;
        h->n_eval = h->n;
    }
    return SPH_OK;
}

int sph_synchronize(sph_handle *h) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    return check_flags(h);
}

int sph_host_register(void *ptr, int64_t bytes) {
    if (!ptr || bytes <= 0) return fail(SPH_ERR_ARG, "bad pointer or size");
    CUDA_TRY(cudaHostRegister(ptr, (size_t)bytes, cudaHostRegisterDefault));
    return SPH_OK;
}

int sph_host_unregister(void *ptr) {
    if (!ptr) return fail(SPH_ERR_ARG, "bad pointer");
    CUDA_TRY(cudaHostUnregister(ptr));
    return SPH_OK;
}

int sph_host_alloc(int64_t bytes, void **ptr) {
    if (!ptr || bytes <= 0) return fail(SPH_ERR_ARG, "bad pointer or size");
    *ptr = nullptr;
    CUDA_TRY(cudaHostAlloc(ptr, (size_t)bytes, cudaHostAllocDefault));
    return SPH_OK;
}

int sph_host_free(void *ptr) {
    if (!ptr) return fail(SPH_ERR_ARG, "bad pointer");
    CUDA_TRY(cudaFreeHost(ptr));
    return SPH_OK;
}

int sph_step_timed(sph_handle *h, int32_t nsteps, double *ms) {
    if (!h || nsteps < 0 || !ms) return fail(SPH_ERR_ARG, "bad argument");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_step_timed before sph_upload");
    int rc = ensure_graphs(h);
    if (rc) return rc;
    if (!h->ev[0])
        for (auto &e : h->ev) CUDA_TRY(cudaEventCreate(&e));
    CUDA_TRY(cudaEventRecord(h->ev[0], h->stream));
    for (int32_t s = 0; s < nsteps; s++) {
        if (h->step == 0) CUDA_TRY(cudaGraphLaunch(h->g_init, h->stream));
        CUDA_TRY(cudaGraphLaunch(h->g_step, h->stream));
        h->step++;
    }
    CUDA_TRY(cudaEventRecord(h->ev[SPH_NUM_STAGES], h->stream));
    CUDA_TRY(cudaEventSynchronize(h->ev[SPH_NUM_STAGES]));
    float t = 0.f;
    CUDA_TRY(cudaEventElapsedTime(&t, h->ev[0], h->ev[SPH_NUM_STAGES]));
    *ms = t;
    if (nsteps > 0) {
        h->evaluated = true;
        h->n_eval = h->n;
    }
    return check_flags(h);
}

int sph_step_profiled(sph_handle *h, int32_t nsteps, double stage_ms[SPH_NUM_STAGES]) {
    if (!h || nsteps < 1 || !stage_ms) return fail(SPH_ERR_ARG, "bad argument");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_step_profiled before sph_upload");
    int rc = ensure_graphs(h);
    if (rc) return rc;
    if (!h->ev[0])
        for (auto &e : h->ev) CUDA_TRY(cudaEventCreate(&e));
    if (!h->g_prof && (rc = capture(h, PRED_DRIFT, true, &h->g_prof, true))) return rc;
    for (int i = 0; i < SPH_NUM_STAGES; i++) stage_ms[i] = 0.0;
    for (int32_t s = 0; s < nsteps; s++) {
        if (h->step == 0) CUDA_TRY(cudaGraphLaunch(h->g_init, h->stream));
        CUDA_TRY(cudaGraphLaunch(h->g_prof, h->stream));
        h->step++;
        CUDA_TRY(cudaStreamSynchronize(h->stream));
        for (int i = 0; i < SPH_NUM_STAGES; i++) {
            float t = 0.f;
            CUDA_TRY(cudaEventElapsedTime(&t, h->ev[i], h->ev[i + 1]));
            stage_ms[i] += t / nsteps;
        }
    }
    h->evaluated = true;
    h->n_eval = h->n;
    return check_flags(h);
}

int32_t sph_kernels_per_step(sph_handle *h) {
    if (!h) return -1;
    Guard g(h);
    if (!h->g_step && ensure_graphs(h)) return -1;
    return h->kernels_per_step;
}

int sph_para_ramp(uint8_t *rgba) {
    if (!rgba) return fail(SPH_ERR_ARG, "null buffer");
    para_ramp_table(rgba);
    return SPH_OK;
}

int sph_set_draw_keys(sph_handle *h, const int64_t *z) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (z) h->zkeys.assign(z, z + h->n);
    else h->zkeys.clear();
    h->zrank_dirty = true;
    return SPH_OK;
}

int sph_render(sph_handle *h, int32_t width, int32_t height, uint8_t *rgba) {
    if (!h || !rgba || width < 1 || height < 1 || width > 16384 || height > 16384)
        return fail(SPH_ERR_ARG, "bad handle, buffer or frame size (1..16384 pixels per side)");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "sph_render before sph_upload");
    if (h->nsims != 1) return fail(SPH_ERR_ARG, "frames are drawn for a single simulation");
    const int64_t npix = (int64_t)width * height;
    if (h->rank_cap < h->cap_n) {
        dfree(h, h->d_zrank);
        dfree(h, h->d_rslot);
        h->d_zrank = h->d_rslot = nullptr;
        if (dalloc(h, &h->d_zrank, h->cap_n) || dalloc(h, &h->d_rslot, h->cap_n))
            return fail(SPH_ERR_NOMEM, "frame buffers");
        h->rank_cap = h->cap_n;
        h->zrank_dirty = true;
        unsigned char lut[256 * 4];
        para_ramp_table(lut);
        if (set_ramp(lut)) return fail(SPH_ERR_CUDA, "colour table upload failed");
    }
    if (h->fb_cap < npix) {
        dfree(h, h->d_fb);
        dfree(h, h->d_rgba);
        h->d_fb = nullptr;
        h->d_rgba = nullptr;
        if (dalloc(h, &h->d_fb, npix) || dalloc(h, &h->d_rgba, npix)) return fail(SPH_ERR_NOMEM, "frame buffers");
        h->fb_cap = npix;
    }
    const int64_t n = h->n;
    if (!h->zkeys.empty() && (int64_t)h->zkeys.size() != n)
        return fail(SPH_ERR_STATE, "draw keys do not match the particle count");
    if (!h->zkeys.empty() && h->zrank_dirty) {
        // painting order: descending Z (the reference sorts by -Z), ties by caller index
        std::vector<int32_t> order((size_t)n), rank((size_t)n);
        for (int64_t i = 0; i < n; i++) order[(size_t)i] = (int32_t)i;
        const std::vector<int64_t> &z = h->zkeys;
        std::sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return z[a] > z[b] || (z[a] == z[b] && a < b); });
        for (int64_t r = 0; r < n; r++) rank[(size_t)order[(size_t)r]] = (int32_t)r;
        CUDA_TRY(cudaMemcpyAsync(h->d_zrank, rank.data(), n * sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
        CUDA_TRY(cudaStreamSynchronize(h->stream));
        h->zrank_dirty = false;
    }
    launch_render(h->ctx(), h->launch(), h->A, h->zkeys.empty() ? nullptr : h->d_zrank, h->d_rslot, h->d_fb,
                  h->D.rho, h->evaluated ? h->n_eval : 0, h->params[0].mass, width, height, h->d_rgba);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(rgba, h->d_rgba, npix * 4, cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

int sph_set_search(sph_handle *h, int32_t tiles) {
    if (!h || (tiles != 0 && tiles != 1 && tiles != 2 && tiles != 4 && tiles != 8))
        return fail(SPH_ERR_ARG, "bad handle or search path");
    Guard g(h);
    const int bdef = default_block_warps(h->k);
    if ((tiles == 4 || tiles == 8) && tiles > bdef)
        return fail(SPH_ERR_ARG, "no block tiles of that many warps for this k");
    h->search_default = false;
    const int tile = tiles ? 1 : 0;
    const int block = tiles == 1 ? bdef : tiles == 2 ? 0 : tiles == 0 ? h->tune.block_warps : tiles;
    if (h->tune.tile != tile || h->tune.block_warps != block) {
        h->tune.tile = tile;
        h->tune.block_warps = block;
        destroy_graphs(h);
    }
    return SPH_OK;
}

int sph_search_stats(sph_handle *h, int64_t *queries, int64_t *deferred) {
    if (!h || !queries || !deferred) return fail(SPH_ERR_ARG, "bad argument");
    Guard g(h);
    int32_t nd = 0;
    if (h->tune.tile && h->evaluated) {
        CUDA_TRY(cudaMemcpyAsync(&nd, h->D.ndefer, sizeof nd, cudaMemcpyDeviceToHost, h->stream));
        CUDA_TRY(cudaStreamSynchronize(h->stream));
    }
    *queries = h->n;
    *deferred = h->tune.tile ? nd : h->n;
    return SPH_OK;
}

int sph_selftest_division(int64_t n, uint64_t seed, int64_t *mismatches) {
    if (!mismatches || n < 0) return fail(SPH_ERR_ARG, "bad argument");
    long long m = 0;
    if (div_selftest(n, seed, &m)) return fail(SPH_ERR_CUDA, "division self-check failed to run");
    *mismatches = m;
    return SPH_OK;
}

int sph_selftest_fp64emu(int64_t n, uint64_t seed, int64_t *mismatches) {
    if (!mismatches || n < 0) return fail(SPH_ERR_ARG, "bad argument");
    long long m = 0;
    if (emu_selftest(n, seed, &m)) return fail(SPH_ERR_CUDA, "fp64 emulation self-check failed to run");
    *mismatches = m;
    return SPH_OK;
}

int sph_probe_peaks(double *fp64_tflops, double *fp32_tflops, double *div_cost, double *sqrt_cost) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return fail(SPH_ERR_CUDA, "no CUDA device available");
    }
    if (probe_peaks(fp64_tflops, fp32_tflops, div_cost, sqrt_cost)) return fail(SPH_ERR_CUDA, "throughput probe failed");
    return SPH_OK;
}

int sph_autotune(sph_handle *h, int32_t use_cache, char *report, int32_t report_len) {
    if (!h) return fail(SPH_ERR_ARG, "null handle");
    Guard g(h);
    if (!h->uploaded || h->step != 0)
        return fail(SPH_ERR_STATE, "sph_autotune runs on a freshly uploaded state (before the first step)");
    const int64_t n = h->n;
    double *d = h->d_io;
    // keep the uploaded state (caller order) to restore it afterwards
    launch_gather_state(h->ctx(), h->launch(), h->A, nullptr, d, d + n, d + 2 * n, d + 3 * n, d + 4 * n, nullptr,
                        nullptr, nullptr);
    CUDA_TRY(cudaGetLastError());
    int rc;
    const KnnTune base = h->tune;
    double ms0 = 0.0;
    if ((rc = apply_levels(h, 0)) || (rc = time_forces(h, 1, &ms0))) return rc;
    // distribution class from the spread of smoothing lengths
    std::vector<double> hs(n);
    CUDA_TRY(cudaMemcpyAsync(hs.data(), h->D.h, n * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    double m1 = 0.0, m2 = 0.0;
    for (double v : hs) { m1 += v; m2 += v * v; }
    m1 /= n;
    const double cv = std::sqrt(std::max(m2 / n - m1 * m1, 0.0)) / std::max(m1, 1e-300);
    const char *dist = cv < 0.2 ? "uniform" : cv < 0.6 ? "mild" : cv < 1.5 ? "clustered" : "extreme";
    const std::string key = tune_key(h, dist);
    TuneChoice best;
    bool cached = use_cache && tune_cache_get(key, &best);
    int trials = 0;
    const int reps = std::max(1, std::min(3, (int)(150.0 / std::max(ms0, 1e-3))));
    if (!cached) {
        // (search path, tile shape, cell side / radius): block tiles of eight
        // or four warps, one tile per warp (theta then only shapes the
        // deferred queries' search), or the per-query search
        const int tiles[] = {1, 1, 1, 0, 0, 0};
        const int blocks[] = {8, 4, 0, 0, 0, 0};
        const float thetas[] = {0.5f, 0.5f, 0.5f, 0.35f, 0.5f, 0.7f};
        const int bdef = default_block_warps(h->k);
        best.ms = 1e300;
        const int dmax = (cv < 0.6) ? 1 : 2;  // clustered data: dense regions want finer cells
        for (int delta = -1; delta <= dmax; delta++) {
            if ((rc = apply_levels(h, delta))) continue;
            for (int v = 0; v < 6; v++) {
                if (blocks[v] > bdef) continue;  // no block kernel with that many warps for this k
                h->tune.tile = tiles[v];
                h->tune.block_warps = blocks[v];
                h->tune.theta = thetas[v];
                h->tune.hgrow = kDefaultHgrow;
                destroy_graphs(h);
                double ms = 0.0;
                if ((rc = time_forces(h, reps, &ms))) return rc;
                trials++;
                if (ms < best.ms) {
                    best.ms = ms;
                    best.theta = thetas[v];
                    best.tile = tiles[v];
                    best.block = blocks[v];
                    best.delta = delta;
                    best.hgrow = kDefaultHgrow;
                }
            }
        }
        if ((rc = apply_levels(h, best.delta))) return rc;
        h->tune.theta = best.theta;
        h->tune.tile = best.tile;
        h->tune.block_warps = best.block;
        // The radius guess's growth factor stays at 1.04: the trials time the
        // uploaded state, on which no smoothing length changes between
        // evaluations, so they favour a tighter guess (1.02) that leaves many
        // more queries to the per-query search once the flow moves (clustered
        // N = 4.19M after 30 steps, mixed kNN stage 1.45 ms at 1.02, 1.22 ms
        // at 1.04, 1.27 ms at 1.06).
        tune_cache_put(key, best);
    }
    h->tune = base;
    h->search_default = false;
    h->tune.theta = best.theta;
    h->tune.hgrow = best.hgrow;
    h->tune.tile = best.tile;
    h->tune.block_warps = best.block;
    if ((rc = apply_levels(h, best.delta))) return rc;
    // back to the uploaded state
    launch_scatter_state(h->ctx(), h->launch(), h->A, nullptr, d, d + n, d + 2 * n, d + 3 * n, d + 4 * n, nullptr, nullptr,
                         nullptr, true);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    h->evaluated = false;
    if (report && report_len > 0) {
        std::ostringstream o;
        o << "{\"key\": \"" << key << "\", \"cached\": " << (cached ? "true" : "false") << ", \"trials\": " << trials
          << ", \"theta\": " << best.theta << ", \"hgrow\": " << best.hgrow << ", \"level_delta\": " << best.delta
          << ", \"tiles\": " << best.tile << ", \"block_warps\": " << best.block
          << ", \"ms_per_eval\": " << best.ms << ", \"ms_default\": " << ms0 << ", \"h_cv\": " << cv
          << ", \"cache\": \"" << tune_cache_path() << "\"}";
        strncpy(report, o.str().c_str(), (size_t)report_len - 1);
        report[report_len - 1] = 0;
    }
    return SPH_OK;
}

// ---- checkpoint / resume: header, then the state arrays in storage order
namespace {
constexpr uint32_t kCkptVersion = 3;

struct CkptHeader {
    char magic[8];      // "SPHGPUCK"
    uint32_t version;   // kCkptVersion
    uint32_t mode;
    int64_t n;
    int32_t nsims, k, step, level_delta;
    uint64_t params_hash;
    float theta, hgrow;  // search shape (the mixed form's sums follow its visiting order)
    int32_t tile, block_warps;  // search path (group tiles or per query) and tile shape
    uint64_t payload_hash;  // FNV-1a of the state arrays as stored
};

uint64_t fnv1a(const void *p, size_t len, uint64_t hsh = 1469598103934665603ull) {
    const unsigned char *b = (const unsigned char *)p;
    for (size_t i = 0; i < len; i++) { hsh ^= b[i]; hsh *= 1099511628211ull; }
    return hsh;
}

uint64_t params_hash(const sph_handle *h) {
    uint64_t x = fnv1a(h->params.data(), h->params.size() * sizeof(sph_params));
    return fnv1a(h->offs.data(), h->offs.size() * sizeof(int64_t), x);
}

struct ArrayRef {
    void *dev;
    size_t bytes;
};

std::vector<ArrayRef> state_arrays(sph_handle *h) {
    const size_t n = (size_t)h->n;
    const PArrays &A = h->A;
    return {{A.pos, 16 * n}, {A.vel, 16 * n}, {A.vp, 16 * n}, {A.acc, 16 * n}, {A.u, 8 * n},
            {A.up, 8 * n},   {A.udot, 8 * n}, {A.id, 4 * n},  {A.hprev, 4 * n}};
}

// A checkpoint's payload is checked on the host before anything reaches the
// device: the kernels index the caller's order by `id` (gathers write rho[id],
// neighbour lists, diagnostics), so ids outside a simulation's own slot range
// would become out-of-bounds device writes. Checked: the payload hash, that
// the ids of every simulation are a permutation of its slot range, finite
// non-negative previous smoothing lengths (the search's radius guess) and a
// valid search shape.
int check_checkpoint(const sph_handle *h, const CkptHeader &hd, const std::vector<std::vector<char>> &bufs) {
    uint64_t ph = 1469598103934665603ull;
    for (const std::vector<char> &b : bufs) ph = fnv1a(b.data(), b.size(), ph);
    if (ph != hd.payload_hash) return fail(SPH_ERR_ARG, "checkpoint payload does not match its hash (corrupt file)");
    const int64_t n = h->n;
    const int32_t *id = (const int32_t *)bufs[7].data();
    const float *hprev = (const float *)bufs[8].data();
    std::vector<unsigned char> seen((size_t)n, 0);
    for (int s = 0; s < h->nsims; s++)
        for (int64_t i = h->offs[s]; i < h->offs[s + 1]; i++) {
            const int64_t v = id[i];
            if (v < h->offs[s] || v >= h->offs[s + 1] || seen[(size_t)v])
                return fail(SPH_ERR_ARG, "checkpoint particle ids are not a permutation of each simulation's range");
            seen[(size_t)v] = 1;
        }
    for (int64_t i = 0; i < n; i++)
        if (!(hprev[i] >= 0.f && hprev[i] < 3.0e38f)) return fail(SPH_ERR_ARG, "checkpoint smoothing lengths invalid");
    if (!(hd.theta > 0.f && hd.theta < 64.f) || !(hd.hgrow > 0.f && hd.hgrow < 64.f) || (hd.tile != 0 && hd.tile != 1) ||
        (hd.block_warps != 0 && hd.block_warps != 4 && hd.block_warps != 8) ||
        hd.block_warps > default_block_warps(h->k) ||
        hd.level_delta < -kMaxLevel || hd.level_delta > kMaxLevel || hd.step < 0)
        return fail(SPH_ERR_ARG, "checkpoint search settings out of range");
    return SPH_OK;
}
}  // namespace

int sph_save(sph_handle *h, const char *path) {
    if (!h || !path) return fail(SPH_ERR_ARG, "null argument");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "nothing to save before sph_upload");
    CkptHeader hd;
    memset(&hd, 0, sizeof hd);
    memcpy(hd.magic, "SPHGPUCK", 8);
    hd.version = kCkptVersion;
    hd.mode = (uint32_t)h->mode;
    hd.n = h->n;
    hd.nsims = h->nsims;
    hd.k = h->k;
    hd.step = h->step;
    hd.level_delta = h->level_delta;
    hd.params_hash = params_hash(h);
    hd.theta = h->tune.theta;
    hd.hgrow = h->tune.hgrow;
    hd.tile = h->tune.tile;
    hd.block_warps = h->tune.block_warps;
    const std::vector<ArrayRef> arrays = state_arrays(h);
    std::vector<std::vector<char>> bufs(arrays.size());
    uint64_t ph = 1469598103934665603ull;
    for (size_t i = 0; i < arrays.size(); i++) {
        bufs[i].resize(arrays[i].bytes);
        CUDA_TRY(cudaMemcpyAsync(bufs[i].data(), arrays[i].dev, arrays[i].bytes, cudaMemcpyDeviceToHost, h->stream));
        CUDA_TRY(cudaStreamSynchronize(h->stream));
        ph = fnv1a(bufs[i].data(), bufs[i].size(), ph);
    }
    hd.payload_hash = ph;
    std::ofstream f(path, std::ios::binary | std::ios::trunc);
    if (!f) return fail(SPH_ERR_ARG, std::string("cannot write ") + path);
    f.write((const char *)&hd, sizeof hd);
    for (const std::vector<char> &b : bufs) f.write(b.data(), (std::streamsize)b.size());
    if (!f) return fail(SPH_ERR_ARG, std::string("write failed: ") + path);
    return SPH_OK;
}

int sph_load(sph_handle *h, const char *path) {
    if (!h || !path) return fail(SPH_ERR_ARG, "null argument");
    Guard g(h);
    std::ifstream f(path, std::ios::binary);
    if (!f) return fail(SPH_ERR_ARG, std::string("cannot read ") + path);
    CkptHeader hd;
    f.read((char *)&hd, sizeof hd);
    if (!f || memcmp(hd.magic, "SPHGPUCK", 8) != 0 || hd.version != kCkptVersion)
        return fail(SPH_ERR_ARG, "not a version-3 SPH checkpoint");
    if (hd.n != h->n || hd.nsims != h->nsims || hd.k != h->k || hd.mode != (uint32_t)h->mode ||
        hd.params_hash != params_hash(h))
        return fail(SPH_ERR_ARG, "checkpoint was written by a handle with other parameters or sizes");
    // read the whole payload first: a truncated file leaves the handle untouched
    int rc;
    const std::vector<ArrayRef> arrays = state_arrays(h);
    std::vector<std::vector<char>> bufs(arrays.size());
    for (size_t i = 0; i < arrays.size(); i++) {
        bufs[i].resize(arrays[i].bytes);
        f.read(bufs[i].data(), (std::streamsize)arrays[i].bytes);
        if (!f) return fail(SPH_ERR_ARG, "truncated checkpoint");
    }
    if ((rc = check_checkpoint(h, hd, bufs))) return rc;
    if (hd.level_delta != h->level_delta && (rc = apply_levels(h, hd.level_delta))) return rc;
    // the saved run's search: a choice of its own, or (the settings do not tell an
    // equal choice apart) the default, which then goes on following the count
    h->search_default = hd.tile == (default_per_query(h->n, h->mode) ? 0 : 1) &&
                        hd.block_warps == default_block_warps(h->k) && hd.theta == kDefaultTheta &&
                        hd.hgrow == kDefaultHgrow && hd.level_delta == 0;
    if (hd.theta != h->tune.theta || hd.hgrow != h->tune.hgrow || hd.tile != h->tune.tile ||
        hd.block_warps != h->tune.block_warps) {
        h->tune.theta = hd.theta;
        h->tune.hgrow = hd.hgrow;
        h->tune.tile = hd.tile;
        h->tune.block_warps = hd.block_warps;
        destroy_graphs(h);
    }
    for (size_t i = 0; i < arrays.size(); i++)
        CUDA_TRY(cudaMemcpyAsync(arrays[i].dev, bufs[i].data(), arrays[i].bytes, cudaMemcpyHostToDevice, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    h->step = hd.step;
    h->uploaded = true;
    h->evaluated = false;
    return SPH_OK;
}

int32_t sph_current_step(const sph_handle *h) { return h ? h->step : -1; }
int64_t sph_num_particles(const sph_handle *h) { return h ? h->n : -1; }

int sph_diagnostics(sph_handle *h, int32_t sim, double out[4]) {
    if (!h || !out) return fail(SPH_ERR_ARG, "null argument");
    Guard g(h);
    if (!h->uploaded) return fail(SPH_ERR_STATE, "no state uploaded");
    if (sim >= h->nsims) return fail(SPH_ERR_ARG, "simulation index out of range");
    int64_t lo = sim < 0 ? 0 : h->offs[sim], hi = sim < 0 ? h->n : h->offs[sim + 1];
    launch_diagnostics(h->ctx(), h->launch(), h->A, h->D, lo, hi, h->d_io);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(out, h->d_io + 3 * h->n + 3 * 64, 4 * sizeof(double), cudaMemcpyDeviceToHost,
                             h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

}  // extern "C"
