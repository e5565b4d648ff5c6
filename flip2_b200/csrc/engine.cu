// engine.cu -- the flip_engine handle: the B200 counterpart of the
// reference's Particles class (engine/particles.hu:11-95, particles.cu).
//
// Ownership: the handle owns every device buffer.  Buffers whose size is
// known at flip_create/flip_set_domain come from one arena allocation; the
// reference-mode voxel buffers, whose size depends on the particles, grow
// geometrically and are never shrunk (the reference reallocates with
// cudaMallocAsync every step).  Nothing is allocated inside flip_step in
// native mode.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "common.cuh"
#include "lprec.cuh"
#include "mg.cuh"
#include "native.cuh"
#include "ref_kernels.cuh"

using namespace flip;

struct flip_engine {
    flip_params P{};
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    uint64_t n = 0;
    bool have_domain = false, binned = false, have_voxels = false;
    flip_grid grid{};
    std::string err;

    // arena
    char* arena = nullptr;
    size_t arena_bytes = 0;

    // shared binning buffers
    uint32_t *keys = nullptr, *perm = nullptr, *flags = nullptr, *starts = nullptr, *node_keys = nullptr;
    uint32_t* d_counts = nullptr;  // [0] nodes/tiles, [1] grid tiles, [2] speed bits, [4] device error word, rest spare
    // d_counts + 4: the look-back timeout bit of every sort and scan this
    // engine runs accumulates here; read at the host sync points below
    uint32_t* d_err = nullptr;
    uint32_t err_seen = 0;         // device error bits reported so far (flip_get_info)
    void* sort_scratch = nullptr;
    size_t sort_scratch_bytes = 0;
    void* scan_scratch = nullptr;
    size_t scan_scratch_bytes = 0;
    int key_bits = 32;
    uint32_t* h_small = nullptr;  // pinned readback words
    uint32_t nodes = 0;

    // ---- reference mode (FP64)
    double* pd[6] = {};  // px py pz vx vy vz
    double* pt[6] = {};  // gather targets
    uint32_t *ytable = nullptr, *counts = nullptr, *masks = nullptr, *node_voxels = nullptr;
    uint64_t node_cap = 0;
    double *getmax_n = nullptr, *getmax_vox = nullptr;  // block maxima of particle and of voxel arrays
    uint64_t vox_cap = 0;
    uint32_t voxels = 0;
    uint32_t* voxel_ids = nullptr;
    int8_t* solids = nullptr;
    double *ux = nullptr, *uy = nullptr, *uz = nullptr, *divU = nullptr, *p = nullptr, *res = nullptr;
    double dt = 0.0, frameDt = 1.0 / 24.0, elapsed = 0.0, elapsedThisFrame = 0.0, residual = 0.0;
    uint32_t gs_iters = 0;

    // ---- native mode (FP32)
    NatDims D{};
    uint64_t nslots = 0, ntiles_total = 0;
    float* fp[6] = {};
    float* fq[6] = {};
    float *m[3] = {}, *w[3] = {}, *o[3] = {};
    // x-fastest copies of the projected (ulin) and P2G (olin) face velocities:
    // the grids G2P stages by TMA, through the descriptors in g2p_maps
    float *ulin[3] = {}, *olin[3] = {};
    NatG2PMaps g2p_maps{};
    // keys[p] holds the tile key of particle p's current position (G2P writes
    // them for the next step; uploads invalidate them)
    bool keys_valid = false;
    uint32_t* head_dense = nullptr;  // first particle of each tile key (segment heads of the native binning)
    // captured steps and frames (native mode): the device keeps the solve's
    // outcome (d_rec) and the sub-step control (d_frame); step_graph and
    // frame_graph are rebuilt when the domain, the solids or the solve
    // configuration change
    SolveRecord* d_rec = nullptr;
    FrameState* d_frame = nullptr;
    SolveRecord* h_rec = nullptr;        // pinned readback of d_rec
    FrameState* h_frame = nullptr;       // pinned readback of d_frame
    bool rec_pending = false;            // d_rec is newer than the host's copy of the last solve
    uint64_t rec_chunks_counted[2] = {0, 0};
    uint64_t rec_fallbacks_counted = 0;
    cudaGraphExec_t step_graph = nullptr, frame_graph = nullptr;
    uint32_t step_graph_launches = 0;   // kernels of one captured step outside its loops
    float* cap_fp0 = nullptr;           // fp[0] when the graphs were captured (eager steps swap fp and fq)
    bool cap_off = false;               // capturing failed here: steps run launch by launch
    uint64_t graph_steps = 0;           // steps run as graph launches (flip_info)
    static constexpr int kCapStreams = 4;
    cudaStream_t cap_streams[kCapStreams] = {};
    int cap_depth = 0;
    uint8_t *type = nullptr, *solid_tiled = nullptr, *tile_flags = nullptr;
    bool has_solid = false;
    float usolid[3] = {0.0f, 0.0f, 0.0f};  // velocity of the interior solid cells (native)
    uint32_t* grid_tiles = nullptr;
    PcgBuffers pcg{};
    uint8_t* cell_prev = nullptr;  // cell codes of the previous step's solve (warm start)
    bool warm_ok = false;          // pcg.x holds the previous step's converged pressure
    PcgState* h_state = nullptr;
    cudaGraphExec_t pcg_graph = nullptr;
    int pcg_graph_iters = 0, pcg_graph_limit = 0;
    int sms = 148;
    int last_iters = 0, last_converged = 0;
    double last_rel = 0.0;
    flip_solve_info last_solve{};
    // learned preconditioner: weights survive flip_set_domain, the
    // activation buffers are per domain and allocated on first use
    LpNet lp{};
    char* lp_warena = nullptr;   // w, g, m, v, wb
    char* lp_aarena = nullptr;   // act[3], actz[3], gact, gact2, z, f0, xs, ev, scalars
    float* lp_f0 = nullptr;      // f(0) of the current problem's geometry
    double* lp_scalar = nullptr; // [0..2] m.Am, m.r, e.r; [3] r.r sum
    float* lp_xs = nullptr;      // reference solution of the current problem (training)
    float* lp_ev = nullptr;      // error sample e with A e = r
    bool xstar_ready = false;    // lp_xs holds the current problem's solution
    bool solution_fresh = false; // pcg.x + pcg.xg is a converged solution of the current problem
    uint64_t noise_counter = 0;
    bool lp_have_weights = false;
    cudaGraphExec_t fpcg_graph = nullptr;
    int fpcg_graph_iters = 0, fpcg_graph_limit = 0;
    // multilevel preconditioner (pressure_method 2): levels per domain,
    // allocated on first use; level 0 is the solver's grid
    MgHierarchy mg{};
    char* mg_arena = nullptr;
    float* mg_zn = nullptr;      // network output on the coarsest level
    float* mg_ev = nullptr;      // coarsest error sample (training)
    float* mg_wbuf = nullptr;    // A m - r of the training loss
    float* mg_gz = nullptr;      // dL/dN on the coarsest level
    float* mg_s[3] = {};         // scratch of the coarsest CG
    int* mg_iters = nullptr;     // iterations of the coarsest CG
    cudaGraphExec_t mg_graph = nullptr;
    int mg_graph_iters = 0, mg_graph_limit = 0, mg_graph_coarse = -1;
    bool poisson_ready = false;  // a standalone pressure problem is in place
    float4* gen_sph = nullptr;   // generator inputs (device)
    float* gen_imp = nullptr;
    cudaEvent_t solve_ev[2] = {};
    // streamed round trips (flip_step_streamed_f32): copy streams and the
    // events that order each chunk's upload after the previous download
    static constexpr int kRtChunks = 8;
    cudaStream_t up_stream = nullptr, down_stream = nullptr;
    cudaEvent_t ev_down[kRtChunks] = {}, ev_start = nullptr, ev_up = nullptr, ev_step = nullptr;
    bool rt_down_pending = false;
    uint32_t launches = 0;
    // stage timing
    bool timing = false;
    cudaEvent_t ev[FLIP_NUM_STAGES + 1] = {};
    double stage_ms[FLIP_NUM_STAGES] = {};
    int mark(int k) {
        if (!timing) return FLIP_OK;
        return cuda(cudaEventRecord(ev[k], stream), "cudaEventRecord");
    }

    int fail(int code, const std::string& what) {
        err = what;
        set_error_text(what.c_str());
        return code;
    }
    int cuda(cudaError_t e, const char* what) {
        if (e == cudaSuccess) return FLIP_OK;
        int c = set_cuda_error(e, what);
        err = error_text();
        return c;
    }
};

#define E_TRY(expr)                                            \
    do {                                                       \
        int _r = (expr);                                       \
        if (_r != FLIP_OK) {                                   \
            if (e->err.empty()) e->err = ::flip::error_text(); \
            return _r;                                         \
        }                                                      \
    } while (0)
#define E_CUDA(expr) E_TRY(e->cuda((expr), #expr))

static size_t al(size_t v) { return (v + 255) / 256 * 256; }
constexpr int kGenMaxSpheres = 4096;
constexpr int kGenMaxImpulses = 64;

// Work on the engine stream that follows a streamed round trip must not
// touch the particle buffers while that call's download still reads them:
// order the engine stream after the download (a device-side wait).
static int rt_join(flip_engine* e) {
    if (!e->rt_down_pending) return FLIP_OK;
    E_CUDA(cudaStreamWaitEvent(e->stream, e->ev_down[flip_engine::kRtChunks - 1], 0));
    e->rt_down_pending = false;
    return FLIP_OK;
}

// The engine's device error word: dev_err_fetch queues its copy into the
// pinned readback area before a synchronisation the caller makes anyway;
// dev_err_eval, after that synchronisation, turns a set bit into
// FLIP_ERR_TIMEOUT (and clears the word for the next call).
static int dev_err_fetch(flip_engine* e) {
    return e->cuda(cudaMemcpyAsync(e->h_small + 4, e->d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, e->stream),
                   "cudaMemcpyAsync(error word)");
}
static int dev_err_eval(flip_engine* e) {
    const uint32_t w = e->h_small[4];
    if (!w) return FLIP_OK;
    e->h_small[4] = 0;
    e->err_seen |= w;
    E_CUDA(cudaMemsetAsync(e->d_err, 0, sizeof(uint32_t), e->stream));
    return e->fail(FLIP_ERR_TIMEOUT, (w & DEVERR_TMA_TIMEOUT)
                                         ? "a TMA copy of G2P timed out; the particles of this step are invalid"
                                     : (w & DEVERR_GRID_TIMEOUT)
                                         ? "a grid-wide reduction of the pressure solve timed out; the pressure of this "
                                           "step is invalid"
                                         : "a decoupled look-back wait of the sort or scan timed out; the binning of "
                                           "this step is invalid");
}
static int dev_err_check(flip_engine* e) {
    E_TRY(dev_err_fetch(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    return dev_err_eval(e);
}

extern "C" void flip_default_params(int mode, flip_params* out) {
    if (!out) return;
    memset(out, 0, sizeof(*out));
    out->mode = mode;
    out->flip_ratio = 0.95f;
    out->gravity_y = -9.8f;
    out->pcg_tol = 1e-6;
    out->pcg_max_iter = 5000;
    out->pcg_check_every = 16;
    out->true_residual_every = 64;
    out->permute_velocities = 0;
    out->device = 0;
    out->max_substep_dt = 1.0 / 240.0;
    out->pressure_method = 0;
    out->learned_max_iter = 100;
    out->pcg_warm_start = 1;
}

extern "C" int flip_create(uint64_t n, const flip_params* params, void* stream, flip_engine** out) {
    if (!out || n == 0 || n >= (1ull << 30)) {
        set_error_text("flip_create: n must be in 1..2^30-1 and out non-null");
        return FLIP_ERR_ARG;
    }
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error_text("flip_create: no CUDA device");
        return FLIP_ERR_DEVICE;
    }
    flip_engine* e = new flip_engine();
    if (params) e->P = *params;
    else flip_default_params(FLIP_MODE_NATIVE, &e->P);
    if (e->P.pcg_check_every <= 0) e->P.pcg_check_every = 16;
    if (e->P.max_substep_dt <= 0.0) e->P.max_substep_dt = 1.0 / 240.0;
    e->n = n;
    int rc = e->cuda(cudaSetDevice(e->P.device), "cudaSetDevice");
    if (rc) { delete e; return rc; }
    cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, e->P.device);
    if (stream) {
        e->stream = (cudaStream_t)stream;
    } else {
        rc = e->cuda(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking), "cudaStreamCreate");
        if (rc) { delete e; return rc; }
        e->own_stream = true;
    }
    rc = e->cuda(cudaMallocHost((void**)&e->h_small, 4096), "cudaMallocHost");
    if (rc) { flip_destroy(e); return rc; }
    rc = e->cuda(cudaMallocHost((void**)&e->h_state, sizeof(PcgState)), "cudaMallocHost");
    e->h_rec = reinterpret_cast<SolveRecord*>(reinterpret_cast<char*>(e->h_small) + 256);
    e->h_frame = reinterpret_cast<FrameState*>(reinterpret_cast<char*>(e->h_small) + 512);
    if (rc) { flip_destroy(e); return rc; }
    for (auto& v : e->solve_ev) {
        rc = e->cuda(cudaEventCreate(&v), "cudaEventCreate");
        if (rc) { flip_destroy(e); return rc; }
    }
    *out = e;
    return FLIP_OK;
}

static void free_lp_activations(flip_engine* e) {
    if (e->fpcg_graph) { cudaGraphExecDestroy(e->fpcg_graph); e->fpcg_graph = nullptr; }
    if (e->mg_graph) { cudaGraphExecDestroy(e->mg_graph); e->mg_graph = nullptr; }
    if (e->lp_aarena) cudaFree(e->lp_aarena);
    e->lp_aarena = nullptr;
    for (auto& a : e->lp.act) a = nullptr;
    for (auto& a : e->lp.actz) a = nullptr;
    e->lp_f0 = nullptr;
    e->lp.gact = e->lp.gact2 = nullptr;
    e->pcg.z = nullptr;
    e->lp_scalar = nullptr;
    e->lp.err = nullptr;
    e->lp_xs = e->lp_ev = nullptr;
    e->xstar_ready = false;
}
static void free_mg(flip_engine* e) {
    if (e->mg_graph) { cudaGraphExecDestroy(e->mg_graph); e->mg_graph = nullptr; }
    if (e->mg_arena) cudaFree(e->mg_arena);
    e->mg_arena = nullptr;
    e->mg = MgHierarchy{};
}
static void free_step_graphs(flip_engine* e) {
    if (e->step_graph) { cudaGraphExecDestroy(e->step_graph); e->step_graph = nullptr; }
    if (e->frame_graph) { cudaGraphExecDestroy(e->frame_graph); e->frame_graph = nullptr; }
}
static void free_arena(flip_engine* e) {
    free_step_graphs(e);
    free_mg(e);
    free_lp_activations(e);
    e->poisson_ready = false;
    if (e->pcg_graph) { cudaGraphExecDestroy(e->pcg_graph); e->pcg_graph = nullptr; }
    if (e->arena) cudaFree(e->arena);
    e->arena = nullptr;
    e->arena_bytes = 0;
}
static void free_ref_voxels(flip_engine* e) {
    void* ps[] = {e->voxel_ids, e->solids, e->ux, e->uy, e->uz, e->divU, e->p, e->res, e->getmax_vox};
    for (void* q : ps) if (q) cudaFree(q);
    e->voxel_ids = nullptr; e->solids = nullptr;
    e->ux = e->uy = e->uz = e->divU = e->p = e->res = e->getmax_vox = nullptr;
    e->vox_cap = 0;
}

static int bits_for(uint64_t maxkey) {
    int b = 1;
    while (b < 32 && (maxkey >> b) != 0) ++b;
    return b;
}

extern "C" int flip_set_domain(flip_engine* e, double nx, double ny, double nz, uint32_t x, uint32_t y, uint32_t z,
                               double cellSize) {
    if (!e) return FLIP_ERR_ARG;
    if (x == 0 || y == 0 || z == 0 || !(cellSize > 0.0)) return e->fail(FLIP_ERR_ARG, "flip_set_domain: empty domain");
    E_CUDA(cudaSetDevice(e->P.device));
    E_TRY(rt_join(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    free_arena(e);
    free_ref_voxels(e);
    e->warm_ok = false;
    e->grid.negX = (float)nx; e->grid.negY = (float)ny; e->grid.negZ = (float)nz;  // Grid narrows to float (grid.hpp:118-129)
    e->grid.sizeX = x; e->grid.sizeY = y; e->grid.sizeZ = z;
    e->grid.cellSize = (float)cellSize;
    e->have_domain = true;
    e->binned = e->have_voxels = false;
    const uint64_t n = e->n;
    std::vector<std::pair<void**, size_t>> plan;
    auto add = [&](void** ptr, size_t bytes) { plan.push_back({ptr, bytes}); };
    add((void**)&e->keys, 4 * n);
    add((void**)&e->perm, 4 * n);
    add((void**)&e->starts, 4 * n);
    add((void**)&e->d_counts, 64);
    e->sort_scratch_bytes = flip_sort_pairs_scratch_bytes(n);
    e->scan_scratch_bytes = scan_scratch_bytes(n);
    add(&e->sort_scratch, e->sort_scratch_bytes);
    add(&e->scan_scratch, e->scan_scratch_bytes);
    if (e->P.mode == FLIP_MODE_REFERENCE) {
        // x <= sizeX etc. after the clamp, so keys are bounded by this value
        uint64_t maxkey = (uint64_t)x + (uint64_t)y * x + (uint64_t)z * x * y;
        e->key_bits = maxkey >= 0xFFFFFFFFull ? 32 : bits_for(maxkey);
        e->node_cap = std::min<uint64_t>(n, maxkey + 1);
        add((void**)&e->flags, 4 * n);
        for (int a = 0; a < 6; ++a) { add((void**)&e->pd[a], 8 * n); add((void**)&e->pt[a], 8 * n); }
        add((void**)&e->ytable, 4 * (size_t)y * z);
        add((void**)&e->counts, 4 * e->node_cap);
        add((void**)&e->node_voxels, 4 * e->node_cap);
        add((void**)&e->masks, 64 * e->node_cap);
        add((void**)&e->getmax_n, flip_ref_getmax_scratch_bytes(n));
    } else {
        uint64_t NX = 4ull * x, NY = 4ull * y, NZ = 4ull * z;
        if (NX % 8 || NY % 8 || NZ % 8)
            return e->fail(FLIP_ERR_ARG, "flip_set_domain: native mode needs 4*size to be a multiple of 8 on every axis");
        NatDims& D = e->D;
        D.nx = (int)NX; D.ny = (int)NY; D.nz = (int)NZ;
        D.tx = D.nx / 8; D.ty = D.ny / 8; D.tz = D.nz / 8;
        D.ox = e->grid.negX; D.oy = e->grid.negY; D.oz = e->grid.negZ;
        D.h = e->grid.cellSize / 4.0f;
        D.inv_h = 1.0f / D.h;
        e->ntiles_total = (uint64_t)D.tx * D.ty * D.tz;
        e->nslots = e->ntiles_total * 512;
        if (e->nslots >= (1ull << 32)) return e->fail(FLIP_ERR_ARG, "flip_set_domain: grid above 2^32 voxels");
        e->key_bits = bits_for(e->ntiles_total - 1);
        add((void**)&e->node_keys, 4 * e->ntiles_total);  // occupied tiles, or fluid tiles of a pressure problem
        add((void**)&e->head_dense, 4 * e->ntiles_total);
        add((void**)&e->gen_sph, sizeof(float4) * kGenMaxSpheres);
        add((void**)&e->gen_imp, sizeof(float) * 7 * kGenMaxImpulses);
        for (int a = 0; a < 6; ++a) { add((void**)&e->fp[a], 4 * n); add((void**)&e->fq[a], 4 * n); }
        // what a step clears lies together (clear_grids)
        for (int c = 0; c < 3; ++c) {
            add((void**)&e->m[c], 4 * e->nslots);
            add((void**)&e->w[c], 4 * e->nslots);
        }
        add((void**)&e->type, e->nslots);
        add((void**)&e->pcg.cell, e->nslots);
        add((void**)&e->tile_flags, e->ntiles_total);
        for (int c = 0; c < 3; ++c) {
            add((void**)&e->o[c], 4 * e->nslots);
            add((void**)&e->ulin[c], 4 * e->nslots);
            add((void**)&e->olin[c], 4 * e->nslots);
        }
        add((void**)&e->grid_tiles, 4 * e->ntiles_total);
        float** pv[6] = {&e->pcg.xg, &e->pcg.b, &e->pcg.r, &e->pcg.p0, &e->pcg.p1, &e->pcg.q};
        for (float** q : pv) add((void**)q, 4 * e->nslots);
        add((void**)&e->pcg.x, 8 * e->nslots);
        add((void**)&e->cell_prev, e->nslots);
        add((void**)&e->pcg.tcoord, 4 * e->ntiles_total);
        add((void**)&e->pcg.st, sizeof(PcgState));
        add((void**)&e->d_rec, sizeof(SolveRecord));
        add((void**)&e->d_frame, sizeof(FrameState));
        add((void**)&e->pcg.partials, sizeof(double) * 4 * kPcgBlocks);
        e->pcg.ctas = (uint32_t)std::min<uint64_t>(std::min(e->sms, kResidentMaxCtas), (e->ntiles_total + 3) / 4);
        e->pcg.cluster = false;
        if (e->ntiles_total <= 4ull * e->pcg.ctas) E_TRY(nat_pcg_cluster(e->pcg.ctas, &e->pcg.cluster));
        e->pcg.mail_tiles = (uint32_t)std::min<uint64_t>(e->ntiles_total, kResidentTiles * e->pcg.ctas);
        add((void**)&e->pcg.slots, 8 * kPcgSlotWords * 4 * (size_t)e->pcg.ctas);
        add((void**)&e->pcg.epoch, sizeof(uint32_t));
        add((void**)&e->pcg.far, e->ntiles_total > kResidentNoFar * e->pcg.ctas ? 4 * 768 * (size_t)e->pcg.mail_tiles : 0);
        add((void**)&e->pcg.mail, 8 * 2 * 6 * 64 * (size_t)e->pcg.mail_tiles);
    }
    size_t total = 0;
    for (auto& pr : plan) total += al(pr.second ? pr.second : 1);
    E_CUDA(cudaMalloc((void**)&e->arena, total));
    e->arena_bytes = total;
    size_t off = 0;
    for (auto& pr : plan) { *pr.first = e->arena + off; off += al(pr.second ? pr.second : 1); }
    e->d_err = e->d_counts + 4;
    e->err_seen = 0;
    E_CUDA(cudaMemsetAsync(e->d_counts, 0, 64, e->stream));
    if (e->P.mode == FLIP_MODE_NATIVE) {
        // zero everything once so that stale tiles read as zero
        E_CUDA(cudaMemsetAsync(e->arena, 0, total, e->stream));
        E_CUDA(cudaStreamSynchronize(e->stream));
        E_TRY(nat_make_g2p_maps(e->g2p_maps, e->ulin, e->olin, e->D));
        e->pcg.warm_ok = &e->d_rec->warm_ok;
    }
    e->keys_valid = false;
    return FLIP_OK;
}

// ------------------------------------------------------------- uploads
extern "C" int flip_upload_particles_f64(flip_engine* e, const double* px, const double* py, const double* pz,
                                         const double* vx, const double* vy, const double* vz, uint64_t n) {
    if (!e || !px || !py || !pz) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "upload before setDomain");
    if (n != e->n) return e->fail(FLIP_ERR_ARG, "upload size differs from the engine size");  // cudaVec.cu:90-93 exits here
    const double* src[6] = {px, py, pz, vx, vy, vz};
    if (e->P.mode == FLIP_MODE_REFERENCE) {
        for (int a = 0; a < 6; ++a) {
            if (src[a]) E_CUDA(cudaMemcpyAsync(e->pd[a], src[a], 8 * n, cudaMemcpyDefault, e->stream));
            else E_CUDA(cudaMemsetAsync(e->pd[a], 0, 8 * n, e->stream));
        }
    } else {
        std::vector<float> tmp(n);
        for (int a = 0; a < 6; ++a) {
            if (src[a]) {
                for (uint64_t i = 0; i < n; ++i) tmp[i] = (float)src[a][i];
                E_CUDA(cudaMemcpyAsync(e->fp[a], tmp.data(), 4 * n, cudaMemcpyDefault, e->stream));
                E_CUDA(cudaStreamSynchronize(e->stream));
            } else {
                E_CUDA(cudaMemsetAsync(e->fp[a], 0, 4 * n, e->stream));
            }
        }
    }
    e->binned = e->have_voxels = false;
    e->keys_valid = false;
    return FLIP_OK;
}

extern "C" int flip_upload_particles_f32(flip_engine* e, const float* px, const float* py, const float* pz,
                                         const float* vx, const float* vy, const float* vz, uint64_t n) {
    if (!e || !px || !py || !pz) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "upload before setDomain");
    if (n != e->n) return e->fail(FLIP_ERR_ARG, "upload size differs from the engine size");
    const float* src[6] = {px, py, pz, vx, vy, vz};
    if (e->P.mode == FLIP_MODE_NATIVE) {
        for (int a = 0; a < 6; ++a) {
            if (src[a]) E_CUDA(cudaMemcpyAsync(e->fp[a], src[a], 4 * n, cudaMemcpyDefault, e->stream));
            else E_CUDA(cudaMemsetAsync(e->fp[a], 0, 4 * n, e->stream));
        }
    } else {
        std::vector<double> tmp(n);
        for (int a = 0; a < 6; ++a) {
            if (src[a]) {
                for (uint64_t i = 0; i < n; ++i) tmp[i] = (double)src[a][i];
                E_CUDA(cudaMemcpyAsync(e->pd[a], tmp.data(), 8 * n, cudaMemcpyDefault, e->stream));
                E_CUDA(cudaStreamSynchronize(e->stream));
            } else {
                E_CUDA(cudaMemsetAsync(e->pd[a], 0, 8 * n, e->stream));
            }
        }
    }
    e->binned = e->have_voxels = false;
    e->keys_valid = false;
    return FLIP_OK;
}

extern "C" int flip_download_particles_f32(flip_engine* e, float* px, float* py, float* pz, float* vx, float* vy,
                                           float* vz, uint64_t n) {
    if (!e) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "download before setDomain");
    if (n != e->n) return e->fail(FLIP_ERR_ARG, "download size differs from the engine size");
    float* dst[6] = {px, py, pz, vx, vy, vz};
    if (e->P.mode == FLIP_MODE_NATIVE) {
        for (int a = 0; a < 6; ++a)
            if (dst[a]) E_CUDA(cudaMemcpyAsync(dst[a], e->fp[a], 4 * n, cudaMemcpyDefault, e->stream));
        E_CUDA(cudaStreamSynchronize(e->stream));
    } else {
        std::vector<double> tmp(n);
        for (int a = 0; a < 6; ++a) {
            if (!dst[a]) continue;
            E_CUDA(cudaMemcpyAsync(tmp.data(), e->pd[a], 8 * n, cudaMemcpyDefault, e->stream));
            E_CUDA(cudaStreamSynchronize(e->stream));
            for (uint64_t i = 0; i < n; ++i) dst[a][i] = (float)tmp[i];
        }
    }
    return FLIP_OK;
}

extern "C" int flip_download_particles_f64(flip_engine* e, double* px, double* py, double* pz, double* vx, double* vy,
                                           double* vz, uint64_t n) {
    if (!e) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "download before setDomain");
    if (n != e->n) return e->fail(FLIP_ERR_ARG, "download size differs from the engine size");
    double* dst[6] = {px, py, pz, vx, vy, vz};
    if (e->P.mode == FLIP_MODE_REFERENCE) {
        for (int a = 0; a < 6; ++a)
            if (dst[a]) E_CUDA(cudaMemcpyAsync(dst[a], e->pd[a], 8 * n, cudaMemcpyDefault, e->stream));
        E_CUDA(cudaStreamSynchronize(e->stream));
    } else {
        std::vector<float> tmp(n);
        for (int a = 0; a < 6; ++a) {
            if (!dst[a]) continue;
            E_CUDA(cudaMemcpyAsync(tmp.data(), e->fp[a], 4 * n, cudaMemcpyDefault, e->stream));
            E_CUDA(cudaStreamSynchronize(e->stream));
            for (uint64_t i = 0; i < n; ++i) dst[a][i] = (double)tmp[i];
        }
    }
    return FLIP_OK;
}

extern "C" int flip_set_solid_velocity(flip_engine* e, double ux, double uy, double uz) {
    if (!e) return FLIP_ERR_ARG;
    if (!std::isfinite(ux) || !std::isfinite(uy) || !std::isfinite(uz))
        return e->fail(FLIP_ERR_ARG, "flip_set_solid_velocity: non-finite velocity");
    E_TRY(rt_join(e));
    if (e->stream) E_CUDA(cudaStreamSynchronize(e->stream));  // a captured launch in flight uses the old value
    e->usolid[0] = (float)ux;
    e->usolid[1] = (float)uy;
    e->usolid[2] = (float)uz;
    free_step_graphs(e);  // the captured steps hold the velocity as a kernel argument
    return FLIP_OK;
}

extern "C" int flip_set_solid_mask(flip_engine* e, const uint8_t* mask_host, uint64_t n_voxels) {
    if (!e) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    if (e->P.mode != FLIP_MODE_NATIVE || !e->have_domain) return e->fail(FLIP_ERR_STATE, "solid mask needs a native-mode domain");
    const NatDims& D = e->D;
    if (n_voxels != (uint64_t)D.nx * D.ny * D.nz) return e->fail(FLIP_ERR_ARG, "solid mask size != voxel count");
    if (!e->solid_tiled) E_CUDA(cudaMalloc((void**)&e->solid_tiled, e->nslots));
    uint8_t* lin = nullptr;
    E_CUDA(cudaMalloc((void**)&lin, n_voxels));
    int rc = e->cuda(cudaMemcpyAsync(lin, mask_host, n_voxels, cudaMemcpyDefault, e->stream), "cudaMemcpyAsync");
    if (!rc) rc = nat_launch_mask_to_tiles(lin, D, e->solid_tiled, e->stream);
    if (!rc) rc = e->cuda(cudaStreamSynchronize(e->stream), "cudaStreamSynchronize");
    cudaFree(lin);
    if (rc) return rc;
    e->has_solid = true;
    free_step_graphs(e);
    return FLIP_OK;
}

// ================================================== reference-mode stages
static int ref_check(flip_engine* e) {
    if (!e) return FLIP_ERR_ARG;
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "call before setDomain");
    return FLIP_OK;
}

static int ref_align(flip_engine* e) {
    return ref_launch_keys(e->pd[0], e->pd[1], e->pd[2], e->n, e->grid, e->keys, nullptr, e->stream);
}

static int ref_sort(flip_engine* e) {
    E_TRY(sort_pairs_ex(e->keys, nullptr, e->keys, e->perm, e->n, e->key_bits, e->sort_scratch, e->sort_scratch_bytes,
                        e->stream, e->d_err, kSpinLimit, 0));
    // sortParticles gathers positions only (particles.cu:69-71); velocities
    // keep their order unless permute_velocities is set
    int na = e->P.permute_velocities ? 6 : 3;
    for (int a = 0; a < na; ++a) {
        E_TRY(ref_gather_f64(e->perm, e->n, e->pd[a], e->pt[a], e->stream));
        std::swap(e->pd[a], e->pt[a]);
    }
    e->binned = true;
    return FLIP_OK;
}

static int ensure_voxels(flip_engine* e, uint64_t need) {
    if (need <= e->vox_cap) return FLIP_OK;
    uint64_t cap = std::max<uint64_t>(need + need / 4, 4096);
    E_CUDA(cudaStreamSynchronize(e->stream));
    free_ref_voxels(e);
    E_CUDA(cudaMalloc((void**)&e->voxel_ids, 4 * cap));
    E_CUDA(cudaMalloc((void**)&e->solids, cap));
    double** d[6] = {&e->ux, &e->uy, &e->uz, &e->divU, &e->p, &e->res};
    for (double** q : d) E_CUDA(cudaMalloc((void**)q, 8 * cap));
    E_CUDA(cudaMalloc((void**)&e->getmax_vox, flip_ref_getmax_scratch_bytes(cap)));
    e->vox_cap = cap;
    return FLIP_OK;
}

static int ref_generate_voxels(flip_engine* e) {
    if (!e->binned) return e->fail(FLIP_ERR_STATE, "generateVoxels before sortParticles");
    if (e->n == 0) return e->fail(FLIP_ERR_STATE, "generateVoxels without particles");
    E_TRY(launch_scan(1, e->keys, e->flags, e->n, e->scan_scratch, e->scan_scratch_bytes, e->stream, e->starts, nullptr,
                      e->d_counts, e->d_err, kSpinLimit, 0));
    E_CUDA(cudaMemcpyAsync(e->h_small, e->d_counts, 4, cudaMemcpyDeviceToHost, e->stream));
    E_TRY(dev_err_fetch(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    E_TRY(dev_err_eval(e));
    e->nodes = e->h_small[0];
    if (e->nodes == 0 || e->nodes > e->node_cap) return e->fail(FLIP_ERR_STATE, "node count out of range");
    E_TRY(ref_launch_ydim(e->starts, e->keys, e->nodes, e->grid, e->ytable, e->stream));
    E_TRY(ref_launch_voxel_counts(e->starts, e->keys, e->nodes, e->n, e->pd[0], e->pd[1], e->pd[2], e->grid, e->counts,
                                  e->masks, e->stream));
    E_TRY(launch_scan(0, e->counts, e->node_voxels, e->nodes, e->scan_scratch, e->scan_scratch_bytes, e->stream, nullptr,
                      nullptr, nullptr, e->d_err, kSpinLimit, 0));
    E_CUDA(cudaMemcpyAsync(e->h_small, e->node_voxels + e->nodes - 1, 4, cudaMemcpyDeviceToHost, e->stream));
    E_TRY(dev_err_fetch(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    E_TRY(dev_err_eval(e));
    e->voxels = e->h_small[0];
    E_TRY(ensure_voxels(e, e->voxels));
    E_TRY(ref_launch_voxel_ids(e->keys, e->nodes, e->masks, e->node_voxels, e->grid, e->voxel_ids, e->solids, e->stream));
    E_CUDA(cudaMemsetAsync(e->p, 0, 8 * (size_t)e->voxels, e->stream));
    e->have_voxels = true;
    return FLIP_OK;
}

static int ref_p2g_stage(flip_engine* e) {
    if (!e->have_voxels) return e->fail(FLIP_ERR_STATE, "particleVelToVoxels before generateVoxels");
    return ref_launch_p2g(e->starts, e->keys, e->nodes, e->n, e->pd[0], e->pd[1], e->pd[2], e->pd[3], e->pd[4], e->pd[5],
                          e->node_voxels, e->voxel_ids, e->solids, e->grid, e->ux, e->uy, e->uz, e->stream);
}

// CudaVec<double>::getMax (cudaVec.cu:205-233) with the reference's reduction;
// scratch: flip_ref_getmax_scratch_bytes(n)
static int ref_getmax(flip_engine* e, const double* a, uint64_t n, double* scratch, bool absolute, double* out) {
    double *b0 = scratch, *b1 = scratch + (n / 512 + 2);
    E_TRY(ref_launch_getmax_level(n, a, b0, absolute ? 1 : 0, e->stream));
    for (uint64_t i = n / 512 + 1; i > 1; i = i / 512 + 1) {
        E_TRY(ref_launch_getmax_level(i, b0, b1, absolute ? 1 : 0, e->stream));
        std::swap(b0, b1);
    }
    double v = 0.0;
    E_CUDA(cudaMemcpyAsync(e->h_small, b0, 8, cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    memcpy(&v, e->h_small, 8);
    *out = v;
    return FLIP_OK;
}

static int ref_courant_dt(flip_engine* e, double* dt) {
    double a, b, c;
    E_TRY(ref_getmax(e, e->pd[3], e->n, e->getmax_n, true, &a));
    E_TRY(ref_getmax(e, e->pd[4], e->n, e->getmax_n, true, &b));
    E_TRY(ref_getmax(e, e->pd[5], e->n, e->getmax_n, true, &c));
    double maxVel = std::max(std::fabs(a), std::max(std::fabs(b), std::fabs(c)));
    double voxelSize = (double)e->grid.cellSize / (8.0 - 2.0 * std::floor(2.0));
    *dt = 0.7 * (voxelSize / maxVel);
    return FLIP_OK;
}

static double ref_scale(const flip_engine* e, double dt) {
    double vs = (double)(e->grid.cellSize / 4.0f);
    return dt / (0.014 * vs * vs);
}

// cudaGSiteration (voxelSolveFunctions.cu:391-412): the convergence reads
// happen after iteration 0 and then every 1024 iterations, so the sweeps in
// between run in shared memory in one launch
static int ref_gs_solve(flip_engine* e, double dt, double threshold, uint32_t max_iter, double* out_res, uint32_t* out_it) {
    double maxR = 10.0, prevR = 100.0;
    uint32_t it = 0;
    const double scale = ref_scale(e, dt), w = 1.9;
    while (maxR > threshold && it < max_iter) {
        uint32_t chunk;
        if (it % 1024 == 0) chunk = 1;
        else chunk = 1024 - it % 1024;
        chunk = std::min(chunk, max_iter - it);
        E_TRY(ref_launch_gs(e->nodes, e->node_voxels, e->voxel_ids, e->solids, e->divU, e->p, e->res, scale, w, chunk,
                            e->stream));
        // the iterations inside a chunk never read the residual, and no exit
        // test can fire before the chunk ends except it == max_iter (the chunk
        // is clipped to it)
        uint32_t first = it;
        it += chunk;
        if (first % 1024 == 0) {
            prevR = maxR;
            E_TRY(ref_getmax(e, e->res, e->voxels, e->getmax_vox, true, &maxR));
        }
        if (it == max_iter || (std::fabs(prevR - maxR) < threshold / 1000 && maxR > threshold)) break;
    }
    *out_res = maxR;
    *out_it = it;
    return FLIP_OK;
}

static int ref_pressure(flip_engine* e) {
    if (!e->have_voxels) return e->fail(FLIP_ERR_STATE, "pressureSolve before generateVoxels");
    const double threshold = 0.01;
    const uint32_t maxIterations = 16384;
    double prevTerm = 100.0, term = 0.0;
    double dt;
    E_TRY(ref_courant_dt(e, &dt));
    if (e->frameDt - e->elapsedThisFrame < dt) dt = e->frameDt - e->elapsedThisFrame;
    E_TRY(ref_launch_gravity(e->voxels, e->solids, e->uy, dt, 0, e->stream));
    E_TRY(ref_launch_divergence(e->nodes, e->node_voxels, e->voxel_ids, e->ux, e->uy, e->uz, e->grid, e->ytable, e->starts,
                                e->keys, e->divU, e->stream));
    uint32_t it = 0, total = 0;
    for (;;) {
        E_TRY(ref_gs_solve(e, dt, threshold, maxIterations, &term, &it));
        total += it;
        if (!(prevTerm - term > 0)) break;
        if (term < threshold) break;
        E_TRY(ref_launch_gravity(e->voxels, e->solids, e->uy, dt, 1, e->stream));
        dt /= 2.0;
        E_CUDA(cudaMemsetAsync(e->p, 0, 8 * (size_t)e->voxels, e->stream));
        E_TRY(ref_launch_gravity(e->voxels, e->solids, e->uy, dt, 0, e->stream));
        prevTerm = term;
        E_TRY(ref_launch_divergence(e->nodes, e->node_voxels, e->voxel_ids, e->ux, e->uy, e->uz, e->grid, e->ytable,
                                    e->starts, e->keys, e->divU, e->stream));
    }
    e->dt = dt;
    e->elapsed += dt;
    e->elapsedThisFrame += dt;
    e->residual = term;
    e->gs_iters = total;
    return FLIP_OK;
}

static int ref_update_vel(flip_engine* e) {
    return ref_launch_velocity_update(e->nodes, e->node_voxels, e->voxel_ids, e->solids, e->p, e->ux, e->uy, e->uz,
                                      ref_scale(e, e->dt), e->stream);
}
static int ref_g2p_stage(flip_engine* e) {
    return ref_launch_g2p(e->starts, e->keys, e->nodes, e->n, e->pd[0], e->pd[1], e->pd[2], e->node_voxels, e->voxel_ids,
                          e->ux, e->uy, e->uz, e->grid, e->pd[3], e->pd[4], e->pd[5], e->stream);
}
static int ref_advect_stage(flip_engine* e) {
    return ref_launch_advect(e->n, e->dt, e->pd[0], e->pd[1], e->pd[2], e->pd[3], e->pd[4], e->pd[5], e->stream);
}
static int ref_move_solids_stage(flip_engine* e) {
    E_TRY(ref_launch_move_solids(e->nodes, e->n, e->starts, e->keys, e->pd[0], e->pd[1], e->pd[2], e->node_voxels,
                                 e->voxel_ids, e->solids, e->grid, e->stream));
    return ref_g2p_stage(e);
}

// ===================================================== native-mode step
static int nat_grid(flip_engine* e, int per_sm) { return e->sms * per_sm; }

static int nat_bin(flip_engine* e) {
    E_TRY(e->mark(0));
    if (!e->keys_valid) {  // else the last G2P wrote them
        E_TRY(nat_launch_keys(e->fp[0], e->fp[1], e->fp[2], e->n, e->D, e->keys, e->stream));
        e->launches += 1;
        e->keys_valid = true;
    }
    E_TRY(e->mark(1));
    // the sort's last pass also marks the segment heads in head_dense
    E_TRY(sort_pairs_ex(e->keys, nullptr, e->keys, e->perm, e->n, e->key_bits, e->sort_scratch, e->sort_scratch_bytes,
                        e->stream, e->d_err, kSpinLimit, 0, e->head_dense, (uint32_t)e->ntiles_total));
    E_TRY(e->mark(2));
    E_TRY(nat_launch_gather(e->perm, e->n, (const float* const*)e->fp, e->fq, e->stream));
    for (int a = 0; a < 6; ++a) std::swap(e->fp[a], e->fq[a]);
    E_TRY(e->mark(3));
    E_TRY(nat_launch_segment_heads(e->head_dense, (uint32_t)e->ntiles_total, e->node_keys, e->starts, e->d_counts,
                                   e->stream));
    E_TRY(e->mark(4));
    e->launches += 2 + (uint32_t)((e->key_bits + 7) / 8) + 1 + 1;
    e->binned = true;
    return FLIP_OK;
}

// momentum, weights, types, cell codes and tile flags in one go: they lie
// together in the arena (nine memsets took 27 us of a 32^3 step, one takes 6)
static int clear_grids(flip_engine* e) {
    char* const first = (char*)e->m[0];
    E_CUDA(cudaMemsetAsync(first, 0, (size_t)((char*)e->tile_flags - first) + al(e->ntiles_total), e->stream));
    return FLIP_OK;
}

static int nat_p2g_stage(flip_engine* e, double dt) {
    // keep the last solve's cell codes for the warm start (a copy: the PCG
    // graphs hold the pcg.cell pointer)
    if (e->P.pcg_warm_start && e->warm_ok)
        E_CUDA(cudaMemcpyAsync(e->cell_prev, e->pcg.cell, e->nslots, cudaMemcpyDeviceToDevice, e->stream));
    E_TRY(clear_grids(e));
    E_TRY(e->mark(5));
    E_TRY(nat_launch_p2g(e->node_keys, e->starts, e->d_counts, e->n, (const float* const*)e->fp,
                         (const float* const*)(e->fp + 3), e->D, e->m, e->w, e->type, nat_grid(e, 8), e->stream));
    if (e->has_solid) E_TRY(nat_launch_apply_solids(e->solid_tiled, e->type, e->nslots, e->stream));
    E_TRY(e->mark(6));
    E_TRY(nat_launch_dilate_compact(e->node_keys, e->d_counts, e->D, e->tile_flags, e->grid_tiles, e->d_counts + 1,
                                    nat_grid(e, 2), e->stream));
    E_TRY(nat_launch_tile_coords(e->node_keys, e->d_counts, e->D, e->pcg.tcoord, nat_grid(e, 2), e->stream));
    E_TRY(e->mark(7));
    E_TRY(nat_launch_normalize(e->grid_tiles, e->d_counts + 1, e->D, (float)(e->P.gravity_y * dt), e->m,
                               (const float* const*)e->w, e->o, e->type,
                               make_float3(e->usolid[0], e->usolid[1], e->usolid[2]), nat_grid(e, 4), e->stream, e->ulin,
                               e->olin));
    E_TRY(e->mark(8));
    e->launches += 1 + (e->has_solid ? 1 : 0) + 3 + 1;
    e->have_voxels = true;
    return FLIP_OK;
}

// A whole solve as one graph: a conditional WHILE node whose body is
// `body` (a chunk of iterations and the true-residual check, captured from
// the engine stream) followed by the loop control kernel, which stops the
// loop when the device state says done or after `limit` chunks.  The host
// launches it once per solve and reads the state once at the end.
template <class Body>
static int build_loop_graph(flip_engine* e, Body body, int limit, cudaGraphExec_t* out) {
    cudaGraph_t g = nullptr;
    E_CUDA(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h;
    cudaError_t ce = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault);
    cudaGraphNodeParams cp = {};
    cudaGraphNode_t node = nullptr;
    if (ce == cudaSuccess) {
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        ce = cudaGraphAddNode(&node, g, nullptr, 0, &cp);
    }
    if (ce == cudaSuccess)
        ce = cudaStreamBeginCaptureToGraph(e->stream, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                           cudaStreamCaptureModeThreadLocal);
    if (ce != cudaSuccess) {
        cudaGraphDestroy(g);
        return e->cuda(ce, "conditional loop graph");
    }
    int rc = body();
    if (rc == FLIP_OK) rc = nat_launch_loop_ctl(h, e->pcg.st, limit, e->stream);
    cudaGraph_t captured = nullptr;
    ce = cudaStreamEndCapture(e->stream, &captured);
    if (rc != FLIP_OK || ce != cudaSuccess) {
        cudaGraphDestroy(g);
        return rc != FLIP_OK ? rc : e->cuda(ce, "cudaStreamEndCapture");
    }
    ce = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    E_CUDA(ce);
    return FLIP_OK;
}

static int loop_limit(int max_iter, int chunk) { return (max_iter + chunk - 1) / chunk + 3; }

static int nat_pcg_graph(flip_engine* e, int iters, int max_iter) {
    const int limit = loop_limit(max_iter, iters);
    if (e->pcg_graph && e->pcg_graph_iters == iters && e->pcg_graph_limit == limit) return FLIP_OK;
    if (e->pcg_graph) { cudaGraphExecDestroy(e->pcg_graph); e->pcg_graph = nullptr; }
    E_TRY(build_loop_graph(e, [&]() {
        int rc = FLIP_OK;
        for (int k = 0; k < iters && rc == FLIP_OK; ++k)
            rc = nat_launch_pcgw_iteration(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
        if (rc == FLIP_OK) rc = nat_launch_pcgw_check(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
        return rc;
    }, limit, &e->pcg_graph));
    e->pcg_graph_iters = iters;
    e->pcg_graph_limit = limit;
    return FLIP_OK;
}

// ------------------------------------------------ learned preconditioner
static int lp_alloc_weights(flip_engine* e) {
    if (e->lp_warena) return FLIP_OK;
    const size_t fw = al(sizeof(float) * kLpNumW), bw = al(sizeof(__nv_bfloat16) * kLpNumW);
    E_CUDA(cudaMalloc((void**)&e->lp_warena, 4 * fw + bw));
    E_CUDA(cudaMemsetAsync(e->lp_warena, 0, 4 * fw + bw, e->stream));
    e->lp.w = (float*)e->lp_warena;
    e->lp.g = (float*)(e->lp_warena + fw);
    e->lp.m = (float*)(e->lp_warena + 2 * fw);
    e->lp.v = (float*)(e->lp_warena + 3 * fw);
    e->lp.wb = (__nv_bfloat16*)(e->lp_warena + 4 * fw);
    const int dil[kLpLayers] = {1, 2, 4, 1};
    for (int l = 0; l < kLpLayers; ++l) e->lp.dil[l] = dil[l];
    e->lp.adam_t = 0;
    e->lp.tensor_cores = e->P.lp_cuda_cores ? 0 : 1;
    e->lp.sms = e->sms;
    return FLIP_OK;
}
// activations for every slot of the grid: 3 x 16 BF16 + 2 x 16 FP32 + z
static int lp_alloc_activations(flip_engine* e) {
    if (e->lp_aarena) return FLIP_OK;
    if (e->P.mode != FLIP_MODE_NATIVE) return e->fail(FLIP_ERR_STATE, "learned preconditioner: native mode only");
    const size_t ab = al(e->nslots * 16 * sizeof(__nv_bfloat16)), gb = al(e->nslots * 16 * sizeof(float)),
                 zb = al(e->nslots * sizeof(float));
    const size_t total = 6 * ab + 2 * gb + 4 * zb + 256;
    E_CUDA(cudaMalloc((void**)&e->lp_aarena, total));
    E_CUDA(cudaMemsetAsync(e->lp_aarena, 0, total, e->stream));
    char* q = e->lp_aarena;
    for (int l = 0; l < 3; ++l, q += ab) e->lp.act[l] = (__nv_bfloat16*)q;
    for (int l = 0; l < 3; ++l, q += ab) e->lp.actz[l] = (__nv_bfloat16*)q;
    e->lp.gact = (float*)q; q += gb;
    e->lp.gact2 = (float*)q; q += gb;
    e->pcg.z = (float*)q; q += zb;
    e->lp_f0 = (float*)q; q += zb;
    e->lp_xs = (float*)q; q += zb;
    e->lp_ev = (float*)q; q += zb;
    e->lp_scalar = (double*)q;
    e->lp.err = (int*)(q + 64);
    e->xstar_ready = false;
    return FLIP_OK;
}
// the network's view of the current problem: activations on the dilated
// tile list, outputs on the occupied (fluid) tiles
static LpGrid lp_grid(flip_engine* e, const int* halt) {
    LpGrid G{};
    G.r = e->pcg.r;
    G.type = e->type;
    G.tile_active = e->tile_flags;
    G.act_tiles = e->grid_tiles;
    G.d_nact = e->d_counts + 1;
    G.out_tiles = e->node_keys;
    G.d_nout = e->d_counts;
    G.halt = halt;
    G.cell = e->pcg.cell;
    G.D = e->D;
    return G;
}
// the tensor-core kernels' error word: a bounded wait that gave up
static int lp_check_err(flip_engine* e) {
    if (!e->lp.err) return FLIP_OK;
    int w = 0;
    E_CUDA(cudaMemcpyAsync(&w, e->lp.err, sizeof(int), cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    if (w) return e->fail(FLIP_ERR_TIMEOUT, "learned preconditioner: a tensor-core wait timed out");
    return FLIP_OK;
}
static int lp_ready(flip_engine* e) {
    if (!e->lp_have_weights) return e->fail(FLIP_ERR_STATE, "learned preconditioner: no weights (flip_lp_init or flip_lp_set_weights)");
    return lp_alloc_activations(e);
}

// ------------------------------------------------ multilevel preconditioner
// the hierarchy of the domain: coarse levels allocated once per domain;
// level 0 points at the solver's buffers (pcg.z lives with the network's)
static int mg_ready(flip_engine* e, bool network) {
    if (network) E_TRY(lp_ready(e));
    else E_TRY(lp_alloc_activations(e));
    MgHierarchy& H = e->mg;
    if (!e->mg_arena) {
        MgLevel L[kMgMaxLevels];
        const int levels = mg_plan(e->D.nx, e->D.ny, e->D.nz, e->D.h, L, kMgMaxLevels);
        const size_t fine = (size_t)e->nslots;
        size_t total = al(4 * fine);
        for (int l = 1; l < levels; ++l) {
            const size_t n = (size_t)L[l].ntiles * 512u;
            total += 2 * al(n) + al(L[l].ntiles) + al(4 * (size_t)L[l].ntiles) + 3 * al(4 * n) + 256;
        }
        const size_t nc = (size_t)L[levels - 1].ntiles * 512u;
        total += 8 * al(4 * nc) + 1024 + al(sizeof(double) * kMgScalePartials) + 256;
        E_CUDA(cudaMalloc((void**)&e->mg_arena, total));
        E_CUDA(cudaMemsetAsync(e->mg_arena, 0, total, e->stream));
        char* q = e->mg_arena;
        auto take = [&](size_t b) { char* r = q; q += al(b); return r; };
        L[0].t = (float*)take(4 * fine);
        std::vector<uint32_t> iota;
        for (int l = 1; l < levels; ++l) {
            MgLevel& c = L[l];
            const size_t n = (size_t)c.ntiles * 512u;
            c.type = (uint8_t*)take(n);
            c.cell = (uint8_t*)take(n);
            c.active = (uint8_t*)take(c.ntiles);
            uint32_t* tiles = (uint32_t*)take(4 * (size_t)c.ntiles);
            uint32_t* count = (uint32_t*)take(256);
            c.r = (float*)take(4 * n);
            c.z = (float*)take(4 * n);
            c.t = (float*)take(4 * n);
            c.tiles = tiles;
            c.d_ntiles = count;
            iota.resize(c.ntiles);
            for (uint32_t t = 0; t < c.ntiles; ++t) iota[t] = t;
            E_CUDA(cudaMemcpyAsync(tiles, iota.data(), 4 * (size_t)c.ntiles, cudaMemcpyHostToDevice, e->stream));
            E_CUDA(cudaMemcpyAsync(count, &c.ntiles, 4, cudaMemcpyHostToDevice, e->stream));
            E_CUDA(cudaMemsetAsync(c.active, 1, c.ntiles, e->stream));
            E_CUDA(cudaStreamSynchronize(e->stream));  // iota and ntiles are host locals
        }
        e->mg_zn = (float*)take(4 * nc);
        e->mg_ev = (float*)take(4 * nc);
        e->mg_wbuf = (float*)take(4 * nc);
        e->mg_gz = (float*)take(4 * nc);
        for (auto& p : e->mg_s) p = (float*)take(4 * nc);
        H.f0 = (float*)take(4 * nc);
        H.inv_s = (float*)take(256);
        H.scale_partials = (double*)take(sizeof(double) * kMgScalePartials);
        H.scale_ticket = (unsigned int*)take(256);
        e->mg_iters = (int*)take(256);
        H.levels = levels;
        for (int l = 0; l < levels; ++l) H.L[l] = L[l];
    }
    // level 0: the solver's grid and vectors
    MgLevel& f = H.L[0];
    f.D = e->D;
    f.tiles = e->node_keys;
    f.d_ntiles = e->d_counts;
    f.type = e->type;
    f.cell = e->pcg.cell;
    f.r = e->pcg.r;
    f.z = e->pcg.z;
    f.ntiles = (uint32_t)e->ntiles_total;
    return FLIP_OK;
}
// the network's view of the coarsest level (every tile active)
static LpGrid mg_lp_grid(flip_engine* e, const int* halt) {
    const MgLevel& c = e->mg.L[e->mg.levels - 1];
    if (e->mg.levels == 1) {
        LpGrid G = lp_grid(e, halt);
        G.r = c.r;
        return G;
    }
    LpGrid G{};
    G.r = c.r;
    G.type = c.type;
    G.tile_active = c.active;
    G.act_tiles = c.tiles;
    G.d_nact = c.d_ntiles;
    G.out_tiles = c.tiles;
    G.d_nout = c.d_ntiles;
    G.halt = halt;
    G.cell = c.cell;
    G.D = c.D;
    return G;
}
static int mg_coarse_grid(flip_engine* e) {
    const uint32_t n = e->mg.L[e->mg.levels - 1].ntiles;
    return e->mg.levels == 1 ? nat_grid(e, 2) : (int)std::min<uint32_t>(n, (uint32_t)e->sms * 2u);
}
// the network on the coarsest level: the small-grid kernels when it is a
// coarse level, the solver-grid kernels when the solver's grid is itself the
// coarsest
static int mg_net_bias(flip_engine* e, const LpGrid& G) {
    if (e->mg.levels == 1) return lp_bias_dev(e->lp, G, e->mg.inv_s, e->mg.f0, mg_coarse_grid(e), e->stream);
    return lp_small_bias(e->lp, G, e->mg.L[e->mg.levels - 1].ntiles, e->mg.inv_s, e->mg.f0, e->stream);
}
static int mg_net_forward(flip_engine* e, const LpGrid& G) {
    if (e->mg.levels == 1) return lp_forward_dev(e->lp, G, e->mg.inv_s, e->mg.f0, e->mg_zn, mg_coarse_grid(e), e->stream);
    return lp_small_forward(e->lp, G, e->mg.L[e->mg.levels - 1].ntiles, e->mg.inv_s, e->mg.f0, e->mg_zn, e->stream);
}
// kernels of one V-cycle (for the launch count)
// kernels of one V-cycle; dot: with FCG's dot products (their own kernel
// only when there is no level above the coarsest to fuse them into)
static uint32_t mg_cycle_launches(flip_engine* e, bool network, bool dot = false) {
    // the network's four kernels, and its input scale when no down kernel takes it
    const uint32_t coarse = network ? (e->mg.levels >= 2 ? 4u : 5u) : (e->P.mg_coarse == 2 ? 1u : 0u);
    return 2u * (uint32_t)(e->mg.levels - 1) + 1u + coarse + (dot && e->mg.levels < 2 ? 1u : 0u);
}
// coarse CG of mg_coarse = 2: relative tolerance and iteration cap
constexpr double kMgCoarseCgTol = 1e-3;
constexpr int kMgCoarseCgIters = 64;
// one V-cycle: z = M(r) from pcg.r into pcg.z (halt: stop when the solve is
// done); dot_init >= 0: then FCG's dot products (init: beta = 0), fused into
// level 0's post-smoothing
static int mg_cycle(flip_engine* e, bool network, const int* halt, int dot_init = -1) {
    const int grid0 = nat_grid(e, 4);
    // with the network and a level above the coarsest, the last down kernel
    // also takes the network's input scale
    const bool fused_scale = network && e->mg.levels >= 2;
    E_TRY(mg_down(e->mg, halt, grid0, e->stream, fused_scale));
    const float* zn = nullptr;
    bool solved = false;
    if (network) {
        const LpGrid G = mg_lp_grid(e, halt);
        if (!fused_scale) E_TRY(mg_input_scale(e->mg, halt, e->stream));
        E_TRY(mg_net_forward(e, G));
        zn = e->mg_zn;
    } else if (e->P.mg_coarse == 2) {
        // the classical comparison: Jacobi-PCG on the coarsest level in one CTA
        const MgLevel& c = e->mg.L[e->mg.levels - 1];
        E_TRY(mg_cg(c, c.r, e->mg_zn, e->mg_s[0], e->mg_s[1], e->mg_s[2], kMgCoarseCgTol, kMgCoarseCgIters, e->mg_iters,
                    e->stream, halt));
        zn = e->mg_zn;
        solved = true;
    }
    E_TRY(mg_coarsest(e->mg, zn, halt, e->stream, solved));
    const bool fuse = dot_init >= 0 && e->mg.levels >= 2;
    const MgDot dot{e->pcg.q, e->pcg.st, e->pcg.partials, dot_init};
    E_TRY(mg_up(e->mg, halt, grid0, e->stream, fuse ? &dot : nullptr));
    if (dot_init >= 0 && !fuse) E_TRY(nat_launch_fpcg_dot(e->node_keys, e->d_counts, e->pcg, dot_init, e->stream, 0));
    return FLIP_OK;
}
// per problem: coarse types and codes (after pcg_init set level 0's codes)
// and the network's f(0) on the coarsest level
static int mg_setup_problem(flip_engine* e, bool network) {
    E_TRY(mg_build(e->mg, nullptr, e->stream));
    e->launches += 2u * (uint32_t)(e->mg.levels - 1) + 2u * (uint32_t)std::max(0, e->mg.levels - 2);
    if (network) {
        const LpGrid G = mg_lp_grid(e, nullptr);
        E_TRY(mg_net_bias(e, G));
        e->launches += 4;
    }
    return FLIP_OK;
}

// ------------------------------------------------------ pressure solves
static void pcg_state_host(flip_engine* e, double tol, int max_iter, int flexible) {
    PcgState init{};
    init.tol2 = tol * tol;
    init.max_iter = max_iter;
    init.true_every = e->P.true_residual_every;
    init.next_check = e->P.true_residual_every;
    init.flexible = flexible;
    *e->h_state = init;
}

static int nat_fpcg_graph(flip_engine* e, int iters, int max_iter) {
    const int limit = loop_limit(max_iter, iters);
    if (e->fpcg_graph && e->fpcg_graph_iters == iters && e->fpcg_graph_limit == limit) return FLIP_OK;
    if (e->fpcg_graph) { cudaGraphExecDestroy(e->fpcg_graph); e->fpcg_graph = nullptr; }
    const LpGrid G = lp_grid(e, &e->pcg.st->halt);
    const float* inv_s = &e->pcg.st->inv_s;
    E_TRY(build_loop_graph(e, [&]() {
        int rc = FLIP_OK;
        for (int k = 0; k < iters && rc == FLIP_OK; ++k) {
            rc = nat_launch_fpcg_direction_update(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
            if (rc == FLIP_OK && k == iters - 1)
                rc = nat_launch_pcg_check(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
            if (rc == FLIP_OK) rc = lp_forward_dev(e->lp, G, inv_s, e->lp_f0, e->pcg.z, nat_grid(e, 2), e->stream);
            if (rc == FLIP_OK) rc = nat_launch_fpcg_dot(e->node_keys, e->d_counts, e->pcg, 0, e->stream);
        }
        return rc;
    }, limit, &e->fpcg_graph));
    e->fpcg_graph_iters = iters;
    e->fpcg_graph_limit = limit;
    return FLIP_OK;
}

static int nat_mgpcg_graph(flip_engine* e, int iters, int max_iter, bool network) {
    const int limit = loop_limit(max_iter, iters);
    const int mode = network ? 0 : e->P.mg_coarse;
    if (e->mg_graph && e->mg_graph_iters == iters && e->mg_graph_limit == limit && e->mg_graph_coarse == mode)
        return FLIP_OK;
    if (e->mg_graph) { cudaGraphExecDestroy(e->mg_graph); e->mg_graph = nullptr; }
    const int* halt = &e->pcg.st->halt;
    E_TRY(build_loop_graph(e, [&]() {
        int rc = FLIP_OK;
        for (int k = 0; k < iters && rc == FLIP_OK; ++k) {
            rc = nat_launch_fpcg_direction_update(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
            if (rc == FLIP_OK && k == iters - 1)
                rc = nat_launch_pcg_check(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
            if (rc == FLIP_OK) rc = mg_cycle(e, network, halt, 0);
        }
        return rc;
    }, limit, &e->mg_graph));
    e->mg_graph_iters = iters;
    e->mg_graph_limit = limit;
    e->mg_graph_coarse = mode;
    return FLIP_OK;
}

// one launch of a solve's loop graph; the state comes back once at the end
static int run_loop(flip_engine* e, cudaGraphExec_t g, uint32_t launches_per_chunk) {
    E_CUDA(cudaGraphLaunch(g, e->stream));
    E_CUDA(cudaMemcpyAsync(e->h_state, e->pcg.st, sizeof(PcgState), cudaMemcpyDeviceToHost, e->stream));
    E_TRY(dev_err_fetch(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->launches += (launches_per_chunk + 1u) * (uint32_t)e->h_state->chunks;
    return dev_err_eval(e);
}

// The Jacobi-PCG loop driven from the host, a chunk per launch sequence with
// a state read after each: the same kernels as the loop graph, for profilers
// that do not look inside conditional graph nodes (environment variable
// FLIP2_HOST_SOLVE_LOOP=1; stage timing or the per-stage API only).
static bool host_solve_loop() {
    static const bool on = [] {
        const char* v = std::getenv("FLIP2_HOST_SOLVE_LOOP");
        return v && v[0] == '1';
    }();
    return on;
}
static int run_plain_host(flip_engine* e, int chunk, int max_iter) {
    const int limit = loop_limit(max_iter, chunk);
    for (int c = 0; c < limit; ++c) {
        for (int k = 0; k < chunk; ++k) E_TRY(nat_launch_pcgw_iteration(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
        E_TRY(nat_launch_pcgw_check(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
        E_CUDA(cudaMemcpyAsync(e->h_state, e->pcg.st, sizeof(PcgState), cudaMemcpyDeviceToHost, e->stream));
        E_TRY(dev_err_fetch(e));
        E_CUDA(cudaStreamSynchronize(e->stream));
        e->launches += 2u * (uint32_t)chunk + 1u;
        E_TRY(dev_err_eval(e));
        if (e->h_state->done) break;
    }
    return FLIP_OK;
}

// the resident solve and its state; done = 0: it left the solve to the loop
static int run_resident(flip_engine* e, int chunk, int max_iter) {
    E_TRY(nat_launch_pcg_resident(e->node_keys, e->d_counts, e->D, e->pcg, chunk, loop_limit(max_iter, chunk), e->d_err, e->stream));
    E_CUDA(cudaMemcpyAsync(e->h_state, e->pcg.st, sizeof(PcgState), cudaMemcpyDeviceToHost, e->stream));
    E_TRY(dev_err_fetch(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->launches += 1;
    return dev_err_eval(e);
}

// Solve A x = b on the occupied tiles.  U: face velocities giving b = -div U,
// or nullptr when b is already in pcg.b.  method 1 runs learned FPCG first and,
// if it stops without meeting tol (iteration cap or a non-positive r.z),
// restarts Jacobi-PCG from x = 0.
static int nat_solve(flip_engine* e, const float* const* U, int method, double tol, int max_plain, int max_learned,
                     flip_solve_info* out, bool warm = false) {
    flip_solve_info info{};
    const int chunk = e->P.pcg_check_every;
    const float* const nullU[3] = {nullptr, nullptr, nullptr};
    if (e->timing || out) E_CUDA(cudaEventRecord(e->solve_ev[0], e->stream));
    bool need_plain = true;
    if (method == 2) {
        const bool network = e->P.mg_coarse == 0;
        E_TRY(mg_ready(e, network));
        pcg_state_host(e, tol, max_learned, 1);
        e->h_state->true_every = chunk;
        e->h_state->next_check = chunk;
        E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
        // warm start as for Jacobi-PCG: from the previous step's pressure on
        // the cells fluid in both solves (r = b - A x0 in FP64)
        E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, U ? U : nullU, e->type, e->pcg, e->stream,
                                  warm ? e->cell_prev : nullptr));
        E_TRY(mg_setup_problem(e, network));
        E_TRY(mg_cycle(e, network, &e->pcg.st->halt, 1));
        e->launches += (warm ? 2u : 1u) + mg_cycle_launches(e, network, true);
        E_TRY(e->mark(9));
        E_TRY(nat_mgpcg_graph(e, chunk, max_learned, network));
        E_TRY(run_loop(e, e->mg_graph, (2u + mg_cycle_launches(e, network, true)) * (uint32_t)chunk + 1u));
        E_TRY(nat_launch_solve_record(e->d_rec, e->pcg.st, 1, 0, 0, e->stream));
        E_TRY(lp_check_err(e));
        const PcgState& s = *e->h_state;
        info.iters = s.iter;
        double rr = s.true_checks ? s.rr_true : s.rr;
        info.rel_residual = s.bb > 0.0 ? std::sqrt(rr / s.bb) : 0.0;
        info.converged = s.done == 1;
        need_plain = s.done != 1;
        if (need_plain) { info.fell_back = 1; U = nullptr; }  // b stays in pcg.b
    }
    if (method == 1) {
        E_TRY(lp_ready(e));
        pcg_state_host(e, tol, max_learned, 1);
        // a true-residual check every chunk: FCG gives up when a chunk reduces
        // the residual by less than 10% (device state done = 4)
        e->h_state->true_every = chunk;
        e->h_state->next_check = chunk;
        E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
        E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, U ? U : nullU, e->type, e->pcg, e->stream));
        const LpGrid G = lp_grid(e, &e->pcg.st->halt);
        E_TRY(lp_bias_dev(e->lp, G, &e->pcg.st->inv_s, e->lp_f0, nat_grid(e, 2), e->stream));
        E_TRY(lp_forward_dev(e->lp, G, &e->pcg.st->inv_s, e->lp_f0, e->pcg.z, nat_grid(e, 2), e->stream));
        E_TRY(nat_launch_fpcg_dot(e->node_keys, e->d_counts, e->pcg, 1, e->stream));
        e->launches += 10;
        E_TRY(e->mark(9));
        E_TRY(nat_fpcg_graph(e, chunk, max_learned));
        E_TRY(run_loop(e, e->fpcg_graph, 7u * (uint32_t)chunk + 1u));
        E_TRY(nat_launch_solve_record(e->d_rec, e->pcg.st, 1, 0, 0, e->stream));
        E_TRY(lp_check_err(e));
        const PcgState& s = *e->h_state;
        info.iters = s.iter;
        double rr = s.true_checks ? s.rr_true : s.rr;
        info.rel_residual = s.bb > 0.0 ? std::sqrt(rr / s.bb) : 0.0;
        info.converged = s.done == 1;
        need_plain = s.done != 1;
        if (need_plain) { info.fell_back = 1; U = nullptr; }  // b stays in pcg.b
    }
    if (need_plain) {
        pcg_state_host(e, tol, max_plain, 0);
        E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
        const bool w = warm && method == 0;
        E_TRY(nat_launch_pcgw_init(e->node_keys, e->d_counts, e->grid_tiles, e->d_counts + 1, e->D, U ? U : nullU,
                                   e->type, e->pcg, e->stream, w ? e->cell_prev : nullptr));
        e->launches += w ? 2 : 1;
        if (method == 0) E_TRY(e->mark(9));
        E_TRY(run_resident(e, chunk, max_plain));
        if (e->h_state->done == 0) {  // more tiles than the chip holds
            if (host_solve_loop()) {
                E_TRY(run_plain_host(e, chunk, max_plain));
            } else {
                E_TRY(nat_pcg_graph(e, chunk, max_plain));
                E_TRY(run_loop(e, e->pcg_graph, 2u * (uint32_t)chunk + 1u));
            }
        }
        E_TRY(nat_launch_solve_record(e->d_rec, e->pcg.st, 0, method == 0 ? 0 : 1, 0, e->stream));
        const PcgState& s = *e->h_state;
        if (method != 0) info.plain_iters = s.iter;
        else info.iters = s.iter;
        double rr = s.true_checks ? s.rr_true : s.rr;
        info.rel_residual = s.bb > 0.0 ? std::sqrt(rr / s.bb) : 0.0;
        info.converged = s.done == 1;
    }
    E_TRY(e->mark(10));
    if (e->timing || out) {
        E_CUDA(cudaEventRecord(e->solve_ev[1], e->stream));
        E_CUDA(cudaEventSynchronize(e->solve_ev[1]));
        float ms = 0.0f;
        E_CUDA(cudaEventElapsedTime(&ms, e->solve_ev[0], e->solve_ev[1]));
        info.ms = ms;
    }
    e->last_iters = info.iters + info.plain_iters;
    e->last_converged = info.converged;
    e->solution_fresh = info.converged != 0;
    e->last_rel = info.rel_residual;
    e->last_solve = info;
    if (out) *out = info;
    return FLIP_OK;
}

static int nat_pressure(flip_engine* e) {
    const int learned = e->P.learned_max_iter > 0 ? e->P.learned_max_iter : e->P.pcg_max_iter;
    const bool warm = e->P.pcg_warm_start && e->warm_ok;
    E_TRY(nat_solve(e, (const float* const*)e->m, e->P.pressure_method, e->P.pcg_tol, e->P.pcg_max_iter, learned,
                    e->timing ? &e->last_solve : nullptr, warm));
    e->warm_ok = e->last_converged != 0;
    e->poisson_ready = true;  // b, the cell types and the tile lists of this solve stay in place
    e->xstar_ready = false;
    return FLIP_OK;
}

static int nat_project_stage(flip_engine* e) {
    return nat_launch_project(e->grid_tiles, e->d_counts + 1, e->D, e->pcg.x, e->pcg.xg, e->type, e->m, nat_grid(e, 4),
                              e->stream, e->ulin);
}
// G2P + advection on the tiles of this step's binning; also writes the tile
// key of every new position for the next step's sort
// in and out: the particle state G2P reads (the binning's gathered order)
// and writes; nullptrs mean fp in place.  dt_p: dt from the device.
static int nat_g2p_stage(flip_engine* e, double dt, float* const* in = nullptr, float* const* out = nullptr,
                         const float* dt_p = nullptr) {
    float* const* I = in ? in : e->fp;
    float* const* Q = out ? out : e->fp;
    E_TRY(nat_launch_g2p(e->g2p_maps, e->node_keys, e->starts, e->d_counts, e->n, e->D, (float)dt, e->P.flip_ratio,
                         (const float* const*)e->m, (const float* const*)e->o, (const float* const*)I,
                         (const float* const*)(I + 3), Q, Q + 3, e->keys, e->has_solid ? e->type : nullptr,
                         make_float3(e->usolid[0], e->usolid[1], e->usolid[2]), dt_p, e->d_err, nat_grid(e, 4),
                         e->stream));
    e->keys_valid = true;
    e->binned = false;
    return FLIP_OK;
}

static int rec_refresh(flip_engine* e);
static int nat_step(flip_engine* e, double dt) {
    E_TRY(rec_refresh(e));  // the warm-start flag of a captured step before this one
    E_TRY(nat_bin(e));
    E_TRY(nat_p2g_stage(e, dt));
    E_TRY(nat_pressure(e));
    E_TRY(nat_project_stage(e));
    E_TRY(e->mark(11));
    E_TRY(nat_g2p_stage(e, dt));
    E_TRY(e->mark(12));
    e->launches += 2;
    if (e->timing) {
        E_CUDA(cudaEventSynchronize(e->ev[12]));
        for (int k = 0; k < FLIP_NUM_STAGES; ++k) {
            float ms = 0.0f;
            E_CUDA(cudaEventElapsedTime(&ms, e->ev[k], e->ev[k + 1]));
            e->stage_ms[k] += ms;
        }
    }
    e->dt = dt;
    e->elapsed += dt;
    e->binned = false;
    return FLIP_OK;
}

// ==================================================== captured steps
// A native step, or a whole native frame, as one CUDA graph.  The host
// launches it and reads nothing back: the solve's outcome stays in d_rec
// (read when the caller asks), the warm start follows the device flag
// d_rec->warm_ok, dt and gravity * dt come from d_frame, and conditional
// nodes carry every data-dependent branch -- the solve's iteration loop
// (WHILE), the Jacobi-PCG restart of a flexible solve that missed tol (IF),
// and, for a frame, the loop over Courant-limited sub-steps (WHILE).
// Conditional nodes are added while the stream is being captured; their
// bodies are captured on side streams.
//
// In a captured step the gather writes the sorted state into fq and G2P
// writes the new state back into fp, so that the state always sits in fp
// between launches (the eager path swaps fp and fq instead).

// a conditional handle of the graph being captured on e->stream
static int cap_handle(flip_engine* e, unsigned int dflt, cudaGraphConditionalHandle* h) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaGraph_t g = nullptr;
    E_CUDA(cudaStreamGetCaptureInfo(e->stream, &cs, nullptr, &g, nullptr, nullptr));
    if (cs != cudaStreamCaptureStatusActive) return e->fail(FLIP_ERR_STATE, "conditional handle outside a capture");
    E_CUDA(cudaGraphConditionalHandleCreate(h, g, dflt, cudaGraphCondAssignDefault));
    return FLIP_OK;
}
// add a conditional node on handle h at the capture point of e->stream.  A
// handle's default applies at graph launch only, so a node inside another
// loop's body has its condition set by a kernel before it (cap_loop does).
static int cap_cond_node(flip_engine* e, cudaGraphConditionalNodeType type, cudaGraphConditionalHandle h,
                         cudaGraph_t* body) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    E_CUDA(cudaStreamGetCaptureInfo(e->stream, &cs, nullptr, &g, &deps, &nd));
    if (cs != cudaStreamCaptureStatusActive) return e->fail(FLIP_ERR_STATE, "conditional node outside a capture");
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = type;
    cp.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    E_CUDA(cudaGraphAddNode(&node, g, deps, nd, &cp));
    *body = cp.conditional.phGraph_out[0];
    E_CUDA(cudaStreamUpdateCaptureDependencies(e->stream, &node, 1, cudaStreamSetCaptureDependencies));
    return FLIP_OK;
}
// capture fn() into a conditional body on the next side stream (e->stream
// points at that stream meanwhile, so the launchers record into the body)
template <class Fn>
static int cap_body(flip_engine* e, cudaGraph_t body, Fn fn) {
    if (e->cap_depth >= flip_engine::kCapStreams) return e->fail(FLIP_ERR_STATE, "conditional nodes nested too deep");
    cudaStream_t& side = e->cap_streams[e->cap_depth];
    if (!side) E_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    E_CUDA(cudaStreamBeginCaptureToGraph(side, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    cudaStream_t outer = e->stream;
    e->stream = side;
    e->cap_depth++;
    int rc = fn();
    e->cap_depth--;
    e->stream = outer;
    cudaGraph_t done = nullptr;
    cudaError_t ce = cudaStreamEndCapture(side, &done);
    if (rc != FLIP_OK) return rc;
    E_CUDA(ce);
    return FLIP_OK;
}
// a WHILE loop of chunks: body() then the loop control kernel; the
// condition is set to 1 by a kernel before the node, so the loop also runs
// when it sits inside another loop's body (unless_done: to 0 where that
// state says the solve is done)
template <class Fn>
static int cap_loop(flip_engine* e, int limit, Fn body, const PcgState* unless_done = nullptr) {
    cudaGraphConditionalHandle h;
    cudaGraph_t g = nullptr;
    E_TRY(cap_handle(e, 1u, &h));
    E_TRY(nat_launch_cond_set(h, 1u, e->stream, unless_done));
    E_TRY(cap_cond_node(e, cudaGraphCondTypeWhile, h, &g));
    return cap_body(e, g, [&]() {
        E_TRY(body());
        return nat_launch_loop_ctl(h, e->pcg.st, limit, e->stream);
    });
}
static int cap_plain_chunk(flip_engine* e, int chunk) {
    for (int k = 0; k < chunk; ++k) E_TRY(nat_launch_pcgw_iteration(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
    return nat_launch_pcgw_check(e->node_keys, e->d_counts, e->D, e->pcg, e->stream);
}
static int cap_mg_chunk(flip_engine* e, int chunk, bool network) {
    const int* halt = &e->pcg.st->halt;
    for (int k = 0; k < chunk; ++k) {
        E_TRY(nat_launch_fpcg_direction_update(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
        if (k == chunk - 1) E_TRY(nat_launch_pcg_check(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
        E_TRY(mg_cycle(e, network, halt, 0));
    }
    return FLIP_OK;
}
// the box has no more tiles than the resident solve holds
static bool resident_always(flip_engine* e) {
    return e->ntiles_total <= (uint64_t)kResidentTiles * e->pcg.ctas;
}
// Jacobi-PCG from a fresh state: b from U (nullptr: already in pcg.b),
// warm: from the previous solution where the device flag allows
static int cap_plain_solve(flip_engine* e, const float* const* U, bool warm, int stage) {
    const int chunk = e->P.pcg_check_every;
    const float* const nullU[3] = {nullptr, nullptr, nullptr};
    E_TRY(nat_launch_state_init(e->pcg.st, e->P.pcg_tol, e->P.pcg_max_iter, e->P.true_residual_every, 0, e->stream));
    E_TRY(nat_launch_pcgw_init(e->node_keys, e->d_counts, e->grid_tiles, e->d_counts + 1, e->D, U ? U : nullU, e->type,
                               e->pcg, e->stream, warm ? e->cell_prev : nullptr));
    const int limit = loop_limit(e->P.pcg_max_iter, chunk);
    E_TRY(nat_launch_pcg_resident(e->node_keys, e->d_counts, e->D, e->pcg, chunk, limit, e->d_err, e->stream));
    if (!resident_always(e)) E_TRY(cap_loop(e, limit, [&]() { return cap_plain_chunk(e, chunk); }, e->pcg.st));
    return nat_launch_solve_record(e->d_rec, e->pcg.st, 0, stage, 1, e->stream);
}
// the pressure solve of a captured step (pressure_method 0 or 2)
static int cap_solve(flip_engine* e) {
    const float* const* U = (const float* const*)e->m;
    const bool warm = e->P.pcg_warm_start != 0;
    if (e->P.pressure_method == 0) return cap_plain_solve(e, U, warm, 0);
    const int chunk = e->P.pcg_check_every;
    const int max_learned = e->P.learned_max_iter > 0 ? e->P.learned_max_iter : e->P.pcg_max_iter;
    const bool network = e->P.mg_coarse == 0;
    E_TRY(nat_launch_state_init(e->pcg.st, e->P.pcg_tol, max_learned, chunk, 1, e->stream));
    E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, U, e->type, e->pcg, e->stream,
                              warm ? e->cell_prev : nullptr));
    E_TRY(mg_setup_problem(e, network));
    E_TRY(mg_cycle(e, network, &e->pcg.st->halt, 1));
    E_TRY(cap_loop(e, loop_limit(max_learned, chunk), [&]() { return cap_mg_chunk(e, chunk, network); }));
    E_TRY(nat_launch_solve_record(e->d_rec, e->pcg.st, 1, 0, 1, e->stream));
    // the flexible solve missed tol: Jacobi-PCG restarts from x = 0 on the same b
    cudaGraphConditionalHandle h;
    cudaGraph_t g = nullptr;
    E_TRY(cap_handle(e, 0u, &h));
    E_TRY(nat_launch_fallback_cond(h, e->pcg.st, e->stream));
    E_TRY(cap_cond_node(e, cudaGraphCondTypeIf, h, &g));
    return cap_body(e, g, [&]() { return cap_plain_solve(e, nullptr, false, 1); });
}

static int cap_step(flip_engine* e) {
    const float* dtp = &e->d_frame->dt;
    const float* gdtp = &e->d_frame->gdt;
    // binning (the keys come from the previous G2P or from the launch)
    E_TRY(sort_pairs_ex(e->keys, nullptr, e->keys, e->perm, e->n, e->key_bits, e->sort_scratch, e->sort_scratch_bytes,
                        e->stream, e->d_err, kSpinLimit, 0, e->head_dense, (uint32_t)e->ntiles_total));
    E_TRY(nat_launch_gather(e->perm, e->n, (const float* const*)e->fp, e->fq, e->stream));
    E_TRY(nat_launch_segment_heads(e->head_dense, (uint32_t)e->ntiles_total, e->node_keys, e->starts, e->d_counts,
                                   e->stream));
    // P2G and the face grids
    if (e->P.pcg_warm_start)
        E_CUDA(cudaMemcpyAsync(e->cell_prev, e->pcg.cell, e->nslots, cudaMemcpyDeviceToDevice, e->stream));
    E_TRY(clear_grids(e));
    E_TRY(nat_launch_p2g(e->node_keys, e->starts, e->d_counts, e->n, (const float* const*)e->fq,
                         (const float* const*)(e->fq + 3), e->D, e->m, e->w, e->type, nat_grid(e, 8), e->stream));
    if (e->has_solid) E_TRY(nat_launch_apply_solids(e->solid_tiled, e->type, e->nslots, e->stream));
    E_TRY(nat_launch_dilate_compact(e->node_keys, e->d_counts, e->D, e->tile_flags, e->grid_tiles, e->d_counts + 1,
                                    nat_grid(e, 2), e->stream));
    E_TRY(nat_launch_tile_coords(e->node_keys, e->d_counts, e->D, e->pcg.tcoord, nat_grid(e, 2), e->stream));
    E_TRY(nat_launch_normalize(e->grid_tiles, e->d_counts + 1, e->D, 0.0f, e->m, (const float* const*)e->w, e->o,
                               e->type, make_float3(e->usolid[0], e->usolid[1], e->usolid[2]), nat_grid(e, 4),
                               e->stream, e->ulin, e->olin, gdtp));
    E_TRY(cap_solve(e));
    E_TRY(nat_project_stage(e));
    return nat_g2p_stage(e, 0.0, e->fq, e->fp, dtp);
}
// kernels of one captured step outside its loops and its restart branch
static uint32_t cap_step_launches(flip_engine* e) {
    uint32_t k = 2 + (uint32_t)((e->key_bits + 7) / 8) + 1 + 1;  // sort, gather, heads
    k += 1 + (e->has_solid ? 1 : 0) + 3 + 1;                       // P2G .. normalise
    k += 2 + (e->P.pcg_warm_start ? 1 : 0) + 1;                    // state, init (+ warm), record
    // the resident solve and, where a box may not fit it, its loop's condition
    k += e->P.pressure_method == 0 ? (resident_always(e) ? 1 : 2) : 1;  // method 2: its loop's condition
    if (e->P.pressure_method == 2) {
        const bool network = e->P.mg_coarse == 0;
        k += 2u * (uint32_t)(e->mg.levels - 1) + 2u * (uint32_t)std::max(0, e->mg.levels - 2) + (network ? 4u : 0u);
        k += mg_cycle_launches(e, network, true) + 1;              // first V-cycle, fallback condition
    }
    return k + 2;                                                  // projection, G2P
}

// builds e->step_graph, or e->frame_graph (frame: a WHILE over sub-steps,
// each taking its dt from the device-side Courant rule)
static int cap_build(flip_engine* e, bool frame) {
    if (e->P.pressure_method == 2) E_TRY(mg_ready(e, e->P.mg_coarse == 0));
    // the launchers count, and the G2P stage marks the keys valid, at capture
    // time: both are restored below (the first launch still needs its keys)
    const uint32_t launches = e->launches;
    const bool keys_valid = e->keys_valid;
    cudaGraph_t g = nullptr;
    E_CUDA(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeRelaxed));
    int rc = FLIP_OK;
    if (!frame) {
        rc = cap_step(e);
    } else {
        cudaGraphConditionalHandle h;
        cudaGraph_t body = nullptr;
        rc = cap_handle(e, 1u, &h);
        if (rc == FLIP_OK) rc = cap_cond_node(e, cudaGraphCondTypeWhile, h, &body);
        if (rc == FLIP_OK)
            rc = cap_body(e, body, [&]() {
                E_TRY(nat_launch_vmax(e->n, (const float* const*)(e->fp + 3), e->d_counts + 2, nat_grid(e, 4), e->stream));
                E_TRY(nat_launch_frame_ctl(h, e->d_frame, e->d_counts + 2, e->P.gravity_y, e->stream));
                return cap_step(e);
            });
    }
    cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
    e->launches = launches;
    e->keys_valid = keys_valid;
    if (rc != FLIP_OK) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    E_CUDA(ce);
    e->cap_fp0 = e->fp[0];
    cudaGraphExec_t* out = frame ? &e->frame_graph : &e->step_graph;
    ce = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    E_CUDA(ce);
    e->step_graph_launches = cap_step_launches(e);
    return FLIP_OK;
}
static bool cap_supported(flip_engine* e) {
    return e->P.mode == FLIP_MODE_NATIVE && !e->timing && !e->cap_off &&
           (e->P.pressure_method == 0 || e->P.pressure_method == 2) && e->n > 0;
}
// a graph that cannot be captured or instantiated here (a driver without
// some node type inside conditional bodies, a caller stream that cannot be
// captured) is not an error of the step: the engine keeps stepping launch by
// launch, with the same results
static int cap_build_or_off(flip_engine* e, bool frame) {
    const int rc = cap_build(e, frame);
    if (rc == FLIP_OK) return FLIP_OK;
    free_step_graphs(e);
    e->cap_off = true;
    e->err.clear();
    (void)cudaGetLastError();
    return rc;
}
// before a captured launch: the keys of the current positions, if the last
// G2P did not write them
static int cap_keys(flip_engine* e) {
    if (e->keys_valid) return FLIP_OK;
    E_TRY(nat_launch_keys(e->fp[0], e->fp[1], e->fp[2], e->n, e->D, e->keys, e->stream));
    e->launches += 1;
    e->keys_valid = true;
    return FLIP_OK;
}
static int cap_launched(flip_engine* e, uint32_t steps) {
    e->launches += steps * e->step_graph_launches;
    e->rec_pending = true;
    e->binned = false;
    e->have_voxels = true;
    e->poisson_ready = true;
    e->xstar_ready = false;
    e->solution_fresh = false;
    return FLIP_OK;
}
// one step as a graph launch (no host round trip)
static int nat_step(flip_engine* e, double dt);
static int cap_step_launch(flip_engine* e, double dt) {
    if (e->fp[0] != e->cap_fp0) free_step_graphs(e);
    if (!e->step_graph && cap_build_or_off(e, false) != FLIP_OK) return nat_step(e, dt);
    E_TRY(cap_keys(e));
    E_TRY(nat_launch_step_dt(e->d_frame, dt, e->P.gravity_y, e->stream));
    E_CUDA(cudaGraphLaunch(e->step_graph, e->stream));
    e->launches += 1;
    e->graph_steps += 1;
    E_TRY(cap_launched(e, 1));
    e->dt = dt;
    e->elapsed += dt;
    return FLIP_OK;
}
// the host's copy of the last solve from d_rec (synchronises); also counts
// the loop kernels the captured launches ran
static int rec_refresh(flip_engine* e) {
    if (!e->rec_pending) return FLIP_OK;
    E_CUDA(cudaMemcpyAsync(e->h_rec, e->d_rec, sizeof(SolveRecord), cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    const SolveRecord r = *e->h_rec;
    flip_solve_info info{};
    info.iters = r.iters;
    info.plain_iters = r.plain_iters;
    info.converged = r.converged;
    info.fell_back = r.fell_back;
    info.rel_residual = r.rel_residual;
    e->last_solve = info;
    e->last_iters = r.iters + r.plain_iters;
    e->last_converged = r.converged;
    e->last_rel = r.rel_residual;
    e->warm_ok = r.warm_ok != 0;
    e->solution_fresh = r.converged != 0;
    const int chunk = e->P.pcg_check_every;
    const uint32_t per_plain = 2u * (uint32_t)chunk + 2u;
    uint32_t per_primary = per_plain;
    if (e->P.pressure_method == 2) per_primary = (2u + mg_cycle_launches(e, e->P.mg_coarse == 0, true)) * (uint32_t)chunk + 2u;
    e->launches += (uint32_t)((r.chunks_primary - e->rec_chunks_counted[0]) * per_primary +
                              (r.chunks_plain - e->rec_chunks_counted[1]) * per_plain);
    // a restart runs the state, init, resident (and loop-condition) and record kernels of its branch
    e->launches += (uint32_t)((resident_always(e) ? 4u : 5u) * (r.fallbacks_captured - e->rec_fallbacks_counted));
    e->rec_chunks_counted[0] = r.chunks_primary;
    e->rec_chunks_counted[1] = r.chunks_plain;
    e->rec_fallbacks_counted = r.fallbacks_captured;
    e->rec_pending = false;
    return FLIP_OK;
}

// a whole frame as one graph launch: the device takes sub-steps of
// min(max_substep_dt, 0.7 h / max |v component|, the rest of the frame)
static int eager_frame(flip_engine* e, double frameDt);
static int cap_frame_launch(flip_engine* e, double frame_dt) {
    if (e->fp[0] != e->cap_fp0) free_step_graphs(e);
    if (!e->frame_graph && cap_build_or_off(e, true) != FLIP_OK) return eager_frame(e, frame_dt);
    E_TRY(cap_keys(e));
    E_TRY(nat_launch_frame_init(e->d_frame, frame_dt, e->P.max_substep_dt, (double)e->D.h, e->stream));
    E_CUDA(cudaGraphLaunch(e->frame_graph, e->stream));
    E_CUDA(cudaMemcpyAsync(e->h_frame, e->d_frame, sizeof(FrameState), cudaMemcpyDeviceToHost, e->stream));
    E_TRY(dev_err_fetch(e));
    E_CUDA(cudaStreamSynchronize(e->stream));
    const FrameState f = *e->h_frame;
    e->launches += 2;  // frame init, graph
    e->graph_steps += (uint64_t)f.substeps;
    E_TRY(cap_launched(e, (uint32_t)f.substeps));
    e->launches += 2u * (uint32_t)f.substeps;  // the speed reduction and the sub-step control
    E_TRY(dev_err_eval(e));
    if (f.error) return e->fail(FLIP_ERR_STATE, "solveFrame: dt collapsed");
    e->dt = f.dt;
    e->elapsed += f.t;
    return FLIP_OK;
}

// ============================================================ public API
#define CHECK_E()                                                             \
    do {                                                                      \
        if (!e) return FLIP_ERR_ARG;                                          \
        if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "call before setDomain"); \
        e->err.clear();                                                       \
        E_CUDA(cudaSetDevice(e->P.device));                                   \
        E_TRY(rt_join(e));                                                    \
    } while (0)

extern "C" int flip_align_particles_to_grid(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_align(e);
    E_TRY(nat_launch_keys(e->fp[0], e->fp[1], e->fp[2], e->n, e->D, e->keys, e->stream));
    e->keys_valid = true;
    return FLIP_OK;
}
extern "C" int flip_sort_particles(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_sort(e);
    return nat_bin(e);
}
extern "C" int flip_generate_voxels(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_generate_voxels(e);
    if (!e->binned) E_TRY(nat_bin(e));
    return FLIP_OK;
}
extern "C" int flip_particle_vel_to_voxels(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_p2g_stage(e);
    if (!e->binned) E_TRY(nat_bin(e));
    return nat_p2g_stage(e, e->P.max_substep_dt);
}
extern "C" int flip_pressure_solve(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_pressure(e);
    if (!e->have_voxels) return e->fail(FLIP_ERR_STATE, "pressureSolve before particleVelToVoxels");
    return nat_pressure(e);
}
extern "C" int flip_update_voxel_velocities(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_update_vel(e);
    return nat_project_stage(e);
}
extern "C" int flip_voxel_vels_to_particles(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_g2p_stage(e);
    // native G2P moves the particles as well (advection is fused); it works
    // on the tiles of the current binning
    if (!e->have_voxels) return e->fail(FLIP_ERR_STATE, "voxelVelsToParticles before particleVelToVoxels");
    return nat_g2p_stage(e, e->P.max_substep_dt);
}
extern "C" int flip_advect_particles(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_advect_stage(e);
    return FLIP_OK;  // fused into flip_voxel_vels_to_particles
}
extern "C" int flip_move_solid_particles(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) return ref_move_solids_stage(e);
    return FLIP_OK;  // native mode: G2P clamps into the box and moves particles out of solid cells
}
extern "C" int flip_initialize(flip_engine* e) {
    CHECK_E();
    if (e->P.mode == FLIP_MODE_REFERENCE) {
        E_TRY(ref_align(e));
        E_TRY(ref_sort(e));
        E_TRY(ref_generate_voxels(e));
        E_CUDA(cudaStreamSynchronize(e->stream));
        return FLIP_OK;
    }
    return nat_bin(e);
}
// native Courant limit: 0.7 voxel sizes per sub-step for the fastest velocity
// component, the reference's rule (particles.cu:493-498) on the native voxel;
// 0 when every particle is at rest
static int nat_courant_dt(flip_engine* e, double* dt) {
    E_TRY(nat_launch_vmax(e->n, (const float* const*)(e->fp + 3), e->d_counts + 2, nat_grid(e, 4), e->stream));
    E_CUDA(cudaMemcpyAsync(e->h_small + 2, e->d_counts + 2, sizeof(uint32_t), cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->launches += 1;
    float vmax = 0.0f;
    memcpy(&vmax, e->h_small + 2, sizeof(float));
    *dt = vmax > 0.0f ? 0.7 * (double)e->D.h / (double)vmax : 0.0;
    return FLIP_OK;
}

extern "C" double flip_get_courant_dt(flip_engine* e) {
    if (!e || !e->have_domain) return 0.0;
    double dt = 0.0;
    if (e->P.mode == FLIP_MODE_REFERENCE) {
        if (ref_courant_dt(e, &dt)) return 0.0;
    } else {
        if (cudaSetDevice(e->P.device) != cudaSuccess || nat_courant_dt(e, &dt)) return 0.0;
    }
    return dt;
}

extern "C" int flip_solve_frame(flip_engine* e, double fps) {
    CHECK_E();
    if (!(fps > 0.0)) return e->fail(FLIP_ERR_ARG, "fps must be positive");
    if (e->P.mode == FLIP_MODE_REFERENCE) {
        // Particles::solveFrame (particles.cu:784-803)
        if (!e->have_voxels) return e->fail(FLIP_ERR_STATE, "solveFrame before initialize");
        e->frameDt = 1.0 / fps;
        e->dt = e->frameDt / 10.0;
        e->elapsedThisFrame = 0.0;
        int guard = 0;
        while (e->elapsedThisFrame < e->frameDt) {
            E_TRY(ref_p2g_stage(e));
            E_TRY(ref_pressure(e));
            E_TRY(ref_update_vel(e));
            E_TRY(ref_g2p_stage(e));
            E_TRY(ref_advect_stage(e));
            E_TRY(ref_move_solids_stage(e));
            E_TRY(ref_align(e));
            E_TRY(ref_sort(e));
            E_TRY(ref_generate_voxels(e));
            if (++guard > 1000000) return e->fail(FLIP_ERR_STATE, "solveFrame: dt collapsed");
        }
        return dev_err_check(e);
    }
    const double frameDt = 1.0 / fps;
    if (cap_supported(e)) return cap_frame_launch(e, frameDt);
    return eager_frame(e, frameDt);
}

// a native frame launch by launch: sub-steps of min(max_substep_dt, the
// Courant limit, what is left of the frame), the speed read back per sub-step
static int eager_frame(flip_engine* e, double frameDt) {
    double t = 0.0;
    int guard = 0;
    while (frameDt - t > 1e-12 * frameDt) {
        double dt = std::min(e->P.max_substep_dt, frameDt - t), cfl = 0.0;
        E_TRY(nat_courant_dt(e, &cfl));
        if (cfl > 0.0) dt = std::min(dt, cfl);
        if (!(dt > 1e-9 * frameDt) || ++guard > 100000) return e->fail(FLIP_ERR_STATE, "solveFrame: dt collapsed");
        E_TRY(nat_step(e, dt));
        t += dt;
    }
    return dev_err_check(e);
}

extern "C" int flip_step(flip_engine* e, double dt) {
    CHECK_E();
    if (!(dt > 0.0)) return e->fail(FLIP_ERR_ARG, "dt must be positive");
    if (e->P.mode == FLIP_MODE_NATIVE) return cap_supported(e) ? cap_step_launch(e, dt) : nat_step(e, dt);
    // reference math with a fixed dt: bin, P2G, gravity + divergence, SOR,
    // projection, G2P, advection (no Courant clamp, no dt halving)
    E_TRY(ref_align(e));
    E_TRY(ref_sort(e));
    E_TRY(ref_generate_voxels(e));
    E_TRY(ref_p2g_stage(e));
    E_TRY(ref_launch_gravity(e->voxels, e->solids, e->uy, dt, 0, e->stream));
    E_TRY(ref_launch_divergence(e->nodes, e->node_voxels, e->voxel_ids, e->ux, e->uy, e->uz, e->grid, e->ytable, e->starts,
                                e->keys, e->divU, e->stream));
    double term;
    uint32_t it;
    E_TRY(ref_gs_solve(e, dt, 0.01, 16384, &term, &it));
    e->dt = dt;
    e->residual = term;
    e->gs_iters = it;
    E_TRY(ref_update_vel(e));
    E_TRY(ref_g2p_stage(e));
    E_TRY(ref_advect_stage(e));
    e->elapsed += dt;
    return FLIP_OK;
}

extern "C" int flip_sync(flip_engine* e) {
    if (!e) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));  // the last streamed download, in the engine stream's order
    if (!e->have_domain) {
        E_CUDA(cudaStreamSynchronize(e->stream));
        return FLIP_OK;
    }
    return dev_err_check(e);
}

static int rt_setup(flip_engine* e) {
    if (e->up_stream) return FLIP_OK;
    E_CUDA(cudaStreamCreateWithFlags(&e->up_stream, cudaStreamNonBlocking));
    E_CUDA(cudaStreamCreateWithFlags(&e->down_stream, cudaStreamNonBlocking));
    for (auto& v : e->ev_down) E_CUDA(cudaEventCreateWithFlags(&v, cudaEventDisableTiming));
    E_CUDA(cudaEventCreateWithFlags(&e->ev_start, cudaEventDisableTiming));
    E_CUDA(cudaEventCreateWithFlags(&e->ev_up, cudaEventDisableTiming));
    E_CUDA(cudaEventCreateWithFlags(&e->ev_step, cudaEventDisableTiming));
    return FLIP_OK;
}

// Upload the particle state from host arrays, one native step, and download
// the new state into the same arrays.  The copies run in kRtChunks ranges on
// two copy streams: a range's upload waits only for the previous call's
// download of that range, so one call's download and the next call's upload
// overlap (the host link is full duplex).  Returns before the download ends.
extern "C" int flip_step_streamed_f32(flip_engine* e, float* px, float* py, float* pz, float* vx, float* vy, float* vz,
                                      uint64_t n, double dt) {
    if (!e) return FLIP_ERR_ARG;
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "call before setDomain");
    e->err.clear();
    E_CUDA(cudaSetDevice(e->P.device));
    if (e->P.mode != FLIP_MODE_NATIVE) return e->fail(FLIP_ERR_STATE, "flip_step_streamed_f32: native mode only");
    if (!px || !py || !pz || !vx || !vy || !vz) return e->fail(FLIP_ERR_ARG, "flip_step_streamed_f32: null array");
    if (n != e->n) return e->fail(FLIP_ERR_ARG, "flip_step_streamed_f32: size differs from the engine size");
    if (!(dt > 0.0)) return e->fail(FLIP_ERR_ARG, "dt must be positive");
    E_TRY(rt_setup(e));
    float* host[6] = {px, py, pz, vx, vy, vz};
    const int C = flip_engine::kRtChunks;
    const uint64_t per = (n + C - 1) / C;
    // uploads: after everything already on the engine stream, and range by
    // range after the previous call's download of that range
    E_CUDA(cudaEventRecord(e->ev_start, e->stream));
    E_CUDA(cudaStreamWaitEvent(e->up_stream, e->ev_start, 0));
    for (int c = 0; c < C; ++c) {
        const uint64_t b = std::min<uint64_t>(n, c * per), m = std::min<uint64_t>(n, b + per) - b;
        if (e->rt_down_pending) E_CUDA(cudaStreamWaitEvent(e->up_stream, e->ev_down[c], 0));
        for (int a = 0; a < 6 && m; ++a)
            E_CUDA(cudaMemcpyAsync(e->fp[a] + b, host[a] + b, 4 * m, cudaMemcpyHostToDevice, e->up_stream));
    }
    E_CUDA(cudaEventRecord(e->ev_up, e->up_stream));
    E_CUDA(cudaStreamWaitEvent(e->stream, e->ev_up, 0));
    e->rt_down_pending = false;
    e->binned = e->have_voxels = false;
    e->keys_valid = false;
    E_TRY(cap_supported(e) ? cap_step_launch(e, dt) : nat_step(e, dt));
    // downloads of the new state (the step leaves it in fp)
    E_CUDA(cudaEventRecord(e->ev_step, e->stream));
    E_CUDA(cudaStreamWaitEvent(e->down_stream, e->ev_step, 0));
    for (int c = 0; c < C; ++c) {
        const uint64_t b = std::min<uint64_t>(n, c * per), m = std::min<uint64_t>(n, b + per) - b;
        for (int a = 0; a < 6 && m; ++a)
            E_CUDA(cudaMemcpyAsync(host[a] + b, e->fp[a] + b, 4 * m, cudaMemcpyDeviceToHost, e->down_stream));
        E_CUDA(cudaEventRecord(e->ev_down[c], e->down_stream));
    }
    e->rt_down_pending = true;
    return FLIP_OK;
}

extern "C" int flip_write_positions_csv(flip_engine* e, const char* path) {
    if (!e || !path) return FLIP_ERR_ARG;
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "call before setDomain");
    std::vector<double> x(e->n), y(e->n), z(e->n);
    E_TRY(flip_download_particles_f64(e, x.data(), y.data(), z.data(), nullptr, nullptr, nullptr, e->n));
    FILE* f = fopen(path, "w");
    if (!f) return e->fail(FLIP_ERR_ARG, std::string("cannot open ") + path);
    // std::ostream's default format is %g with 6 significant digits
    for (uint64_t i = 0; i < e->n; ++i) fprintf(f, "%g, %g, %g\n", x[i], y[i], z[i]);
    fclose(f);
    return FLIP_OK;
}

// binary frame: 16-byte header {"FLIP2POS", uint32 count low, uint32 count
// high} then count x 3 float32 (x, y, z interleaved), little endian
extern "C" int flip_write_positions_bin(flip_engine* e, const char* path) {
    if (!e || !path) return FLIP_ERR_ARG;
    if (!e->have_domain) return e->fail(FLIP_ERR_STATE, "call before setDomain");
    std::vector<float> x(e->n), y(e->n), z(e->n), xyz(3 * e->n);
    E_TRY(flip_download_particles_f32(e, x.data(), y.data(), z.data(), nullptr, nullptr, nullptr, e->n));
    for (uint64_t i = 0; i < e->n; ++i) {
        xyz[3 * i] = x[i];
        xyz[3 * i + 1] = y[i];
        xyz[3 * i + 2] = z[i];
    }
    FILE* f = fopen(path, "wb");
    if (!f) return e->fail(FLIP_ERR_ARG, std::string("cannot open ") + path);
    const char magic[8] = {'F', 'L', 'I', 'P', '2', 'P', 'O', 'S'};
    const uint32_t cnt[2] = {(uint32_t)(e->n & 0xFFFFFFFFu), (uint32_t)(e->n >> 32)};
    bool ok = fwrite(magic, 1, 8, f) == 8 && fwrite(cnt, 4, 2, f) == 2 &&
              fwrite(xyz.data(), sizeof(float), xyz.size(), f) == xyz.size();
    ok = (fclose(f) == 0) && ok;
    if (!ok) return e->fail(FLIP_ERR_ARG, std::string("cannot write ") + path);
    return FLIP_OK;
}

extern "C" int flip_get_buffer(flip_engine* e, int which, void** dev_ptr, uint64_t* count, uint32_t* elem_size) {
    if (!e || !dev_ptr || !count || !elem_size) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    const bool ref = e->P.mode == FLIP_MODE_REFERENCE;
    if (!ref && e->have_domain) {  // refresh the device-side tile count
        E_CUDA(cudaMemcpyAsync(e->h_small, e->d_counts, 8, cudaMemcpyDeviceToHost, e->stream));
        E_CUDA(cudaStreamSynchronize(e->stream));
        e->nodes = e->h_small[0];
    }
    if (!ref && which == FLIP_BUF_PRESSURE && e->pcg.x) {
        // the solver keeps the increments since its last true-residual check
        // in the FP32 part xg: hand out the whole solution
        E_TRY(nat_launch_fold_pressure(e->pcg.x, e->pcg.xg, e->pcg.cell, e->nslots, e->stream));
        e->launches += 1;
    }
    void* p = nullptr;
    uint64_t c = 0;
    uint32_t es = 4;
    switch (which) {
    case FLIP_BUF_PX: case FLIP_BUF_PY: case FLIP_BUF_PZ: case FLIP_BUF_VX: case FLIP_BUF_VY: case FLIP_BUF_VZ:
        p = ref ? (void*)e->pd[which] : (void*)e->fp[which];
        c = e->n; es = ref ? 8 : 4; break;
    case FLIP_BUF_KEYS: p = e->keys; c = e->n; break;
    case FLIP_BUF_PERM: p = e->perm; c = e->n; break;
    case FLIP_BUF_FLAGS: p = e->flags; c = ref ? e->n : 0; break;
    case FLIP_BUF_STARTS: p = e->starts; c = e->nodes; break;
    case FLIP_BUF_YTABLE: p = e->ytable; c = ref ? (uint64_t)e->grid.sizeY * e->grid.sizeZ : 0; break;
    case FLIP_BUF_NODE_VOXELS: p = e->node_voxels; c = ref ? e->nodes : 0; break;
    case FLIP_BUF_VOXEL_IDS: p = e->voxel_ids; c = ref ? e->voxels : 0; break;
    case FLIP_BUF_SOLIDS: p = e->solids; c = ref ? e->voxels : 0; es = 1; break;
    case FLIP_BUF_UX: p = ref ? (void*)e->ux : (void*)e->m[0]; c = ref ? e->voxels : e->nslots; es = ref ? 8 : 4; break;
    case FLIP_BUF_UY: p = ref ? (void*)e->uy : (void*)e->m[1]; c = ref ? e->voxels : e->nslots; es = ref ? 8 : 4; break;
    case FLIP_BUF_UZ: p = ref ? (void*)e->uz : (void*)e->m[2]; c = ref ? e->voxels : e->nslots; es = ref ? 8 : 4; break;
    case FLIP_BUF_DIVU: p = ref ? (void*)e->divU : (void*)e->pcg.b; c = ref ? e->voxels : e->nslots; es = ref ? 8 : 4; break;
    case FLIP_BUF_P: p = ref ? (void*)e->p : (void*)e->pcg.x; c = ref ? e->voxels : e->nslots; es = 8; break;
    case FLIP_BUF_RES: p = ref ? (void*)e->res : (void*)e->pcg.r; c = ref ? e->voxels : e->nslots; es = ref ? 8 : 4; break;
    case FLIP_BUF_GRID_U: p = e->m[0]; c = ref ? 0 : e->nslots; break;
    case FLIP_BUF_GRID_V: p = e->m[1]; c = ref ? 0 : e->nslots; break;
    case FLIP_BUF_GRID_W: p = e->m[2]; c = ref ? 0 : e->nslots; break;
    case FLIP_BUF_CELL_TYPE: p = e->type; c = ref ? 0 : e->nslots; es = 1; break;
    case FLIP_BUF_PRESSURE: p = ref ? (void*)e->p : (void*)e->pcg.x; c = ref ? e->voxels : e->nslots; es = 8; break;
    case FLIP_BUF_TILE_LIST: p = e->node_keys; c = ref ? 0 : e->nodes; break;
    case FLIP_BUF_GRID_U_P2G: p = e->o[0]; c = ref ? 0 : e->nslots; break;
    case FLIP_BUF_GRID_V_P2G: p = e->o[1]; c = ref ? 0 : e->nslots; break;
    case FLIP_BUF_GRID_W_P2G: p = e->o[2]; c = ref ? 0 : e->nslots; break;
    case FLIP_BUF_MG_COARSE_TYPE:
    case FLIP_BUF_MG_COARSE_R:
    case FLIP_BUF_MG_COARSE_E: {
        if (ref || !e->mg_arena) break;
        const MgLevel& cl = e->mg.L[e->mg.levels - 1];
        c = (uint64_t)cl.ntiles * 512u;
        if (which == FLIP_BUF_MG_COARSE_TYPE) { p = cl.type; es = 1; }
        else if (which == FLIP_BUF_MG_COARSE_R) p = cl.r;
        else p = e->mg_ev;
        break;
    }
    default: return e->fail(FLIP_ERR_ARG, "unknown buffer id");
    }
    *dev_ptr = p;
    *count = c;
    *elem_size = es;
    return FLIP_OK;
}

extern "C" int flip_read_buffer(flip_engine* e, int which, void* host_dst, uint64_t bytes) {
    if (!e || !host_dst) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    void* p = nullptr;
    uint64_t c = 0;
    uint32_t es = 0;
    E_TRY(flip_get_buffer(e, which, &p, &c, &es));
    if (bytes > c * es || !p) return e->fail(FLIP_ERR_ARG, "flip_read_buffer: more bytes than the buffer holds");
    E_CUDA(cudaMemcpyAsync(host_dst, p, bytes, cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    return FLIP_OK;
}

extern "C" int flip_get_info(flip_engine* e, flip_info* out) {
    if (!e || !out) return FLIP_ERR_ARG;
    E_TRY(rt_join(e));
    if (e->have_domain) E_TRY(rec_refresh(e));
    memset(out, 0, sizeof(*out));
    if (e->have_domain) {
        E_CUDA(cudaStreamSynchronize(e->stream));
        if (e->P.mode == FLIP_MODE_NATIVE) {
            E_CUDA(cudaMemcpy(e->h_small, e->d_counts, 8, cudaMemcpyDeviceToHost));
            e->nodes = e->h_small[0];
            out->nodes = e->h_small[0];
            out->voxels = e->h_small[1];
            out->pressure_iters = e->last_iters;
            out->converged = e->last_converged;
            out->residual = e->last_rel;
            uint32_t ew[2] = {0, 0};
            E_CUDA(cudaMemcpy(ew, e->d_err, 4, cudaMemcpyDeviceToHost));
            if (e->lp.err) E_CUDA(cudaMemcpy(ew + 1, e->lp.err, 4, cudaMemcpyDeviceToHost));
            out->error_flags = e->err_seen | ew[0] | (ew[1] ? 0x4u : 0u);
        } else {
            out->nodes = e->nodes;
            out->voxels = e->voxels;
            out->pressure_iters = (int32_t)e->gs_iters;
            out->converged = e->residual < 0.01 ? 1 : 0;
            out->residual = e->residual;
            uint32_t w = 0;
            E_CUDA(cudaMemcpy(&w, e->d_err, 4, cudaMemcpyDeviceToHost));
            out->error_flags = e->err_seen | w;
        }
    }
    out->dt = e->dt;
    out->elapsed_time = e->elapsed;
    out->n = e->n;
    out->launches = e->launches;
    if (e->have_domain && e->P.mode == FLIP_MODE_NATIVE && e->d_rec) {
        SolveRecord r{};
        E_CUDA(cudaMemcpy(&r, e->d_rec, sizeof(r), cudaMemcpyDeviceToHost));
        out->solves = r.solves;
        out->fallbacks = r.fallbacks;
        out->graph_steps = e->graph_steps;
        out->pressure_iters_total = r.iters_total;
    }
    return FLIP_OK;
}

// ============================== learned preconditioner and pressure problems
namespace {
// splitmix64 (Steele, Lea and Flood, 2014) for the host-side problem generator
struct HostRng {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    double uni() { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }
    double uni(double a, double b) { return a + (b - a) * uni(); }
    double normal() {  // Box-Muller
        double u1 = uni(), u2 = uni();
        if (u1 < 1e-300) u1 = 1e-300;
        return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
    }
};
}  // namespace

#define CHECK_NATIVE(name)                                                                   \
    do {                                                                                     \
        CHECK_E();                                                                           \
        if (e->P.mode != FLIP_MODE_NATIVE) return e->fail(FLIP_ERR_STATE, name ": native mode only"); \
    } while (0)

extern "C" uint64_t flip_lp_num_weights(void) { return (uint64_t)kLpNumW; }

static int lp_upload(flip_engine* e, const float* w) {
    E_CUDA(cudaSetDevice(e->P.device));
    E_TRY(lp_alloc_weights(e));
    E_CUDA(cudaMemcpyAsync(e->lp.w, w, sizeof(float) * kLpNumW, cudaMemcpyHostToDevice, e->stream));
    E_CUDA(cudaMemsetAsync(e->lp.g, 0, sizeof(float) * kLpNumW, e->stream));
    E_CUDA(cudaMemsetAsync(e->lp.m, 0, sizeof(float) * kLpNumW, e->stream));
    E_CUDA(cudaMemsetAsync(e->lp.v, 0, sizeof(float) * kLpNumW, e->stream));
    E_TRY(lp_sync_bf16(e->lp, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->lp.adam_t = 0;
    e->lp_have_weights = true;
    return FLIP_OK;
}

extern "C" int flip_lp_init(flip_engine* e, uint64_t seed) {
    if (!e) return FLIP_ERR_ARG;
    e->err.clear();
    HostRng rng{seed};
    std::vector<float> w(kLpNumW);
    for (int l = 0; l < kLpLayers; ++l) {
        const double sd = std::sqrt(2.0 / (27.0 * kLpCin[l]));  // He-normal over the 27 taps x Cin inputs
        for (int i = kLpWOff[l]; i < kLpWOff[l + 1]; ++i) w[i] = (float)(sd * rng.normal());
    }
    return lp_upload(e, w.data());
}

extern "C" int flip_lp_set_weights(flip_engine* e, const float* w, uint64_t n) {
    if (!e) return FLIP_ERR_ARG;
    e->err.clear();
    if (!w || n != (uint64_t)kLpNumW) return e->fail(FLIP_ERR_ARG, "flip_lp_set_weights: need flip_lp_num_weights() floats");
    for (uint64_t i = 0; i < n; ++i)
        if (!std::isfinite(w[i])) return e->fail(FLIP_ERR_ARG, "flip_lp_set_weights: non-finite weight");
    return lp_upload(e, w);
}

static int lp_download(flip_engine* e, const float* src, float* dst, uint64_t n, const char* name) {
    if (!e) return FLIP_ERR_ARG;
    e->err.clear();
    if (!dst || n != (uint64_t)kLpNumW) return e->fail(FLIP_ERR_ARG, std::string(name) + ": need flip_lp_num_weights() floats");
    if (!e->lp_have_weights) return e->fail(FLIP_ERR_STATE, std::string(name) + ": no weights");
    E_CUDA(cudaSetDevice(e->P.device));
    E_CUDA(cudaMemcpyAsync(dst, src, sizeof(float) * kLpNumW, cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    return FLIP_OK;
}
extern "C" int flip_lp_get_weights(flip_engine* e, float* w, uint64_t n) {
    return lp_download(e, e ? e->lp.w : nullptr, w, n, "flip_lp_get_weights");
}
extern "C" int flip_lp_get_grad(flip_engine* e, float* g, uint64_t n) {
    return lp_download(e, e ? e->lp.g : nullptr, g, n, "flip_lp_get_grad");
}

// fluid tiles -> node_keys, their dilation -> tile_flags / grid_tiles, cell codes cleared
static int poisson_tiles(flip_engine* e) {
    e->warm_ok = false;
    E_CUDA(cudaMemsetAsync(e->pcg.cell, 0, e->nslots, e->stream));
    E_TRY(nat_launch_fluid_tiles(e->type, e->tile_flags, (uint32_t)e->ntiles_total, e->node_keys, e->d_counts, e->nslots,
                                 e->stream));
    E_TRY(nat_launch_dilate_compact(e->node_keys, e->d_counts, e->D, e->tile_flags, e->grid_tiles, e->d_counts + 1,
                                    nat_grid(e, 2), e->stream));
    E_TRY(nat_launch_tile_coords(e->node_keys, e->d_counts, e->D, e->pcg.tcoord, nat_grid(e, 2), e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->launches += 6;
    e->poisson_ready = true;
    e->have_voxels = false;
    e->xstar_ready = false;
    e->solution_fresh = false;
    return FLIP_OK;
}

extern "C" int flip_poisson_generate(flip_engine* e, const flip_poisson_spec* spec) {
    CHECK_NATIVE("flip_poisson_generate");
    if (!spec) return e->fail(FLIP_ERR_ARG, "flip_poisson_generate: null spec");
    if (!(spec->surface_min >= 0.0 && spec->surface_min <= spec->surface_max && spec->surface_max <= 1.0) ||
        !(spec->solid_fraction >= 0.0 && spec->solid_fraction <= 0.5) ||
        !(spec->radius_min > 0.0 && spec->radius_min <= spec->radius_max) || spec->impulses < 0 ||
        spec->impulses > kGenMaxImpulses || !std::isfinite(spec->gravity_dt))
        return e->fail(FLIP_ERR_ARG, "flip_poisson_generate: spec out of range");
    const NatDims& D = e->D;
    HostRng rng{spec->seed};
    const double surface = rng.uni(spec->surface_min, spec->surface_max) * D.ny;
    // spheres until their summed volume reaches the solid fraction of the box
    std::vector<float4> sph;
    const double target = spec->solid_fraction * (double)D.nx * D.ny * D.nz;
    double vol = 0.0;
    while (vol < target && (int)sph.size() < kGenMaxSpheres) {
        const double cx = rng.uni(0.0, D.nx), cy = rng.uni(0.0, D.ny), cz = rng.uni(0.0, D.nz);
        const double r = rng.uni(spec->radius_min, spec->radius_max);
        sph.push_back(make_float4((float)cx, (float)cy, (float)cz, (float)r));
        vol += 4.18879020478639 * r * r * r;
    }
    // Gaussian impulses: centre, width 1/12..1/4 of the smallest extent, N(0,1) amplitudes
    const double ext = std::min(D.nx, std::min(D.ny, D.nz));
    std::vector<float> imp(7 * (size_t)std::max(spec->impulses, 1));
    for (int q = 0; q < spec->impulses; ++q) {
        float* m = imp.data() + 7 * q;
        m[0] = (float)rng.uni(0.0, D.nx);
        m[1] = (float)rng.uni(0.0, D.ny);
        m[2] = (float)rng.uni(0.0, D.nz);
        m[3] = (float)(ext * rng.uni(1.0 / 12.0, 0.25));
        for (int c = 0; c < 3; ++c) m[4 + c] = (float)rng.normal();
    }
    if (!sph.empty())
        E_CUDA(cudaMemcpyAsync(e->gen_sph, sph.data(), sizeof(float4) * sph.size(), cudaMemcpyHostToDevice, e->stream));
    if (spec->impulses > 0)
        E_CUDA(cudaMemcpyAsync(e->gen_imp, imp.data(), sizeof(float) * 7 * spec->impulses, cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_poisson_gen(D, (float)surface, e->gen_sph, (int)sph.size(), e->gen_imp, spec->impulses,
                                 (float)spec->gravity_dt, e->type, e->pcg.b, e->nslots, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));  // the host vectors above are pageable
    e->launches += 1;
    return poisson_tiles(e);
}

extern "C" int flip_poisson_set(flip_engine* e, const uint8_t* type_lin, const float* b_lin) {
    CHECK_NATIVE("flip_poisson_set");
    if (!type_lin || !b_lin) return e->fail(FLIP_ERR_ARG, "flip_poisson_set: null array");
    // pcg.cell and pcg.q stage the linear arrays (nslots == cells)
    E_CUDA(cudaMemcpyAsync(e->pcg.cell, type_lin, e->nslots, cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_mask_to_tiles(e->pcg.cell, e->D, e->type, e->stream));
    E_CUDA(cudaMemcpyAsync(e->pcg.q, b_lin, 4 * e->nslots, cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_lin_tiles_f32(e->pcg.q, e->pcg.b, e->D, 1, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->launches += 2;
    return poisson_tiles(e);
}

extern "C" int flip_poisson_solve(flip_engine* e, int method, double tol, int max_iter, flip_solve_info* info) {
    CHECK_NATIVE("flip_poisson_solve");
    if (!e->poisson_ready) return e->fail(FLIP_ERR_STATE, "flip_poisson_solve: no problem (flip_poisson_generate/set)");
    if (method < 0 || method > 2 || !(tol > 0.0) || max_iter <= 0)
        return e->fail(FLIP_ERR_ARG, "flip_poisson_solve: method 0/1/2, tol > 0, max_iter > 0");
    flip_solve_info local{};
    e->warm_ok = false;  // pcg.x will hold this problem's solution
    const int plain = method != 0 ? e->P.pcg_max_iter : max_iter;
    E_TRY(nat_solve(e, nullptr, method, tol, plain, max_iter, &local));
    if (info) *info = local;
    return FLIP_OK;
}

extern "C" int flip_poisson_read_solution(flip_engine* e, double* x_lin) {
    CHECK_NATIVE("flip_poisson_read_solution");
    if (!x_lin) return e->fail(FLIP_ERR_ARG, "flip_poisson_read_solution: null array");
    double* tmp = nullptr;
    E_CUDA(cudaMalloc((void**)&tmp, 8 * e->nslots));
    int rc = nat_launch_solution_lin(e->pcg.x, e->pcg.xg, e->pcg.cell, e->D, tmp, e->stream);
    if (rc == FLIP_OK) rc = e->cuda(cudaMemcpyAsync(x_lin, tmp, 8 * e->nslots, cudaMemcpyDeviceToHost, e->stream), "cudaMemcpyAsync");
    if (rc == FLIP_OK) rc = e->cuda(cudaStreamSynchronize(e->stream), "cudaStreamSynchronize");
    cudaFree(tmp);
    e->launches += 1;
    return rc;
}

// loss = (m.Am - 2 m.r) / e.r + 1 from the device sums
static int lp_read_loss(flip_engine* e, double* loss) {
    double sums[3] = {0.0, 0.0, 0.0};
    E_CUDA(cudaMemcpyAsync(e->h_small, e->lp_scalar, sizeof(sums), cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    memcpy(sums, e->h_small, sizeof(sums));
    if (loss) *loss = sums[2] > 0.0 ? (sums[0] - 2.0 * sums[1]) / sums[2] + 1.0 : 0.0;
    return FLIP_OK;
}

// the reference solution x* of the current problem, for error samples
static int lp_reference_solution(flip_engine* e) {
    if (e->xstar_ready) return FLIP_OK;
    if (!e->solution_fresh) {
        flip_solve_info info{};
        E_TRY(nat_solve(e, nullptr, 0, e->P.pcg_tol, e->P.pcg_max_iter, e->P.pcg_max_iter, &info));
        if (!info.converged) return e->fail(FLIP_ERR_NOT_CONVERGED, "flip_lp_train_step: the reference solve did not converge");
    }
    const LpGrid G = lp_grid(e, nullptr);
    E_TRY(lp_store_solution(G, e->pcg.x, e->pcg.xg, e->lp_xs, nat_grid(e, 2), e->stream));
    e->launches += 1;
    e->xstar_ready = true;
    return FLIP_OK;
}

// loss, gradient and Adam for the sample in pcg.r / lp_ev (inv_s set)
static int lp_loss_backward(flip_engine* e, const float* inv_s, bool want_grad, float lr, bool step) {
    const LpGrid G = lp_grid(e, nullptr);
    const int grid = nat_grid(e, 2);
    E_TRY(lp_bias_dev(e->lp, G, inv_s, e->lp_f0, grid, e->stream));
    E_TRY(lp_forward_dev(e->lp, G, inv_s, e->lp_f0, e->pcg.z, grid, e->stream));
    E_CUDA(cudaMemsetAsync(e->lp_scalar, 0, 3 * sizeof(double), e->stream));
    E_TRY(lp_loss_grad(G, e->pcg.z, e->lp_ev, e->pcg.q, e->pcg.p1, e->lp_scalar, grid, e->stream));
    e->launches += 8 + 2;
    if (want_grad) {
        E_CUDA(cudaMemsetAsync(e->lp.g, 0, sizeof(float) * kLpNumW, e->stream));
        E_TRY(lp_backward_dev(e->lp, G, inv_s, e->pcg.p1, grid, e->stream));
        e->launches += e->lp.tensor_cores ? 16 : 14;
    }
    if (step) {
        E_TRY(lp_adam(e->lp, lr, e->stream));
        e->launches += 1;
    }
    return FLIP_OK;
}

extern "C" int flip_lp_train_step(flip_engine* e, int sample, float lr, double* loss) {
    CHECK_NATIVE("flip_lp_train_step");
    if (!e->poisson_ready) return e->fail(FLIP_ERR_STATE, "flip_lp_train_step: no problem (flip_poisson_generate/set or a step)");
    if (sample < -1 || sample > 100000 || !(lr >= 0.0f)) return e->fail(FLIP_ERR_ARG, "flip_lp_train_step: bad arguments");
    E_TRY(lp_ready(e));
    E_TRY(lp_reference_solution(e));
    const float* const nullU[3] = {nullptr, nullptr, nullptr};
    const LpGrid G = lp_grid(e, nullptr);
    const int grid = nat_grid(e, 2);
    // pcg_init sets the cell codes, n_fluid, r = b and inv_s = 1/rms(b)
    pcg_state_host(e, 0.0, sample + 1, 0);
    e->h_state->true_every = 0;
    E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, nullU, e->type, e->pcg, e->stream));
    e->launches += 1;
    float* inv_s = &e->pcg.st->inv_s;
    if (sample >= 0) {
        // the residual of x_k after k Jacobi-PCG iterations from 0, and e = x* - x_k
        for (int k = 0; k < sample; ++k) E_TRY(nat_launch_pcg_iteration(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
        E_TRY(lp_error_from_solution(G, e->pcg.x, e->pcg.xg, e->lp_xs, e->lp_ev, grid, e->stream));
        e->launches += 2 * (uint32_t)sample + 1;
    } else {
        // white noise e on the fluid cells and r = A e
        E_TRY(lp_noise_sample(G, 0x5DEECE66Dull + e->noise_counter++, e->lp_ev, e->pcg.r, grid, e->stream));
        E_TRY(lp_input_scale(G, e->lp_scalar + 3, &e->pcg.st->nfluid, inv_s, grid, e->stream));
        e->launches += 4;
    }
    e->solution_fresh = false;  // pcg.x now holds x_k
    e->warm_ok = false;
    E_TRY(lp_loss_backward(e, inv_s, true, lr, true));
    E_TRY(lp_read_loss(e, loss));
    return lp_check_err(e);
}

extern "C" int flip_lp_eval(flip_engine* e, const float* r_lin, const float* e_lin, float* z_lin, double* loss,
                            int want_grad) {
    CHECK_NATIVE("flip_lp_eval");
    if (!e->poisson_ready) return e->fail(FLIP_ERR_STATE, "flip_lp_eval: no problem (flip_poisson_generate/set or a step)");
    if (!r_lin || !e_lin) return e->fail(FLIP_ERR_ARG, "flip_lp_eval: null residual or error");
    E_TRY(lp_ready(e));
    pcg_state_host(e, 0.0, 0, 0);
    E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
    const float* const nullU[3] = {nullptr, nullptr, nullptr};
    E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, nullU, e->type, e->pcg, e->stream));  // cell codes, n_fluid
    e->solution_fresh = false;
    e->warm_ok = false;
    E_CUDA(cudaMemcpyAsync(e->pcg.p0, r_lin, 4 * e->nslots, cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_lin_tiles_f32(e->pcg.p0, e->pcg.r, e->D, 1, e->stream));
    E_CUDA(cudaMemcpyAsync(e->pcg.p0, e_lin, 4 * e->nslots, cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_lin_tiles_f32(e->pcg.p0, e->lp_ev, e->D, 1, e->stream));
    const LpGrid G = lp_grid(e, nullptr);
    float* inv_s = &e->pcg.st->inv_s;
    E_TRY(lp_input_scale(G, e->lp_scalar + 3, &e->pcg.st->nfluid, inv_s, nat_grid(e, 2), e->stream));
    e->launches += 1 + 2 + 2;
    E_TRY(lp_loss_backward(e, inv_s, want_grad != 0, 0.0f, false));
    if (z_lin) {
        E_TRY(nat_launch_lin_tiles_f32(e->pcg.z, e->pcg.p0, e->D, 0, e->stream));
        E_CUDA(cudaMemcpyAsync(z_lin, e->pcg.p0, 4 * e->nslots, cudaMemcpyDeviceToHost, e->stream));
        e->launches += 1;
    }
    E_TRY(lp_read_loss(e, loss));
    return lp_check_err(e);
}

extern "C" int flip_test_solve_timeout(flip_engine* e, int which, uint32_t exchange, uint32_t polls) {
    CHECK_NATIVE("flip_test_solve_timeout");
    if (which < 0 || which > 2 || (exchange && polls < 1024u))
        return e->fail(FLIP_ERR_ARG, "flip_test_solve_timeout: bad arguments");
    E_CUDA(cudaStreamSynchronize(e->stream));
    free_step_graphs(e);  // the captured steps hold one form of the solve's kernel
    e->pcg.hook.which = (uint32_t)which;
    e->pcg.hook.exchange = exchange;
    e->pcg.hook.polls = polls;
    return FLIP_OK;
}

// ------------------------------------------- multilevel preconditioner API
extern "C" int flip_mg_apply(flip_engine* e, const float* r_lin, float* z_lin) {
    CHECK_NATIVE("flip_mg_apply");
    if (!e->poisson_ready) return e->fail(FLIP_ERR_STATE, "flip_mg_apply: no problem (flip_poisson_generate/set or a step)");
    if (!r_lin || !z_lin) return e->fail(FLIP_ERR_ARG, "flip_mg_apply: null residual or output");
    const bool network = e->P.mg_coarse == 0;
    E_TRY(mg_ready(e, network));
    pcg_state_host(e, 0.0, 0, 0);
    E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
    const float* const nullU[3] = {nullptr, nullptr, nullptr};
    E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, nullU, e->type, e->pcg, e->stream));  // cell codes
    e->solution_fresh = false;
    e->warm_ok = false;
    E_CUDA(cudaMemcpyAsync(e->pcg.p0, r_lin, 4 * e->nslots, cudaMemcpyHostToDevice, e->stream));
    E_TRY(nat_launch_lin_tiles_f32(e->pcg.p0, e->pcg.r, e->D, 1, e->stream));
    // the cycle writes the tiles with fluid cells; the others may hold an
    // earlier problem's z
    E_CUDA(cudaMemsetAsync(e->pcg.z, 0, 4 * e->nslots, e->stream));
    E_TRY(mg_setup_problem(e, network));
    E_TRY(mg_cycle(e, network, nullptr));
    E_TRY(nat_launch_lin_tiles_f32(e->pcg.z, e->pcg.p0, e->D, 0, e->stream));
    E_CUDA(cudaMemcpyAsync(z_lin, e->pcg.p0, 4 * e->nslots, cudaMemcpyDeviceToHost, e->stream));
    E_CUDA(cudaStreamSynchronize(e->stream));
    e->launches += 3u + mg_cycle_launches(e, network);
    return lp_check_err(e);
}

extern "C" int flip_mg_train_step(flip_engine* e, int sample, float lr, double* loss) {
    CHECK_NATIVE("flip_mg_train_step");
    if (!e->poisson_ready) return e->fail(FLIP_ERR_STATE, "flip_mg_train_step: no problem (flip_poisson_generate/set or a step)");
    if (sample < -1 || sample > 100000 || !(lr >= 0.0f)) return e->fail(FLIP_ERR_ARG, "flip_mg_train_step: bad arguments");
    E_TRY(mg_ready(e, true));
    pcg_state_host(e, 0.0, sample + 1, 0);
    e->h_state->true_every = 0;
    E_CUDA(cudaMemcpyAsync(e->pcg.st, e->h_state, sizeof(PcgState), cudaMemcpyHostToDevice, e->stream));
    const float* const nullU[3] = {nullptr, nullptr, nullptr};
    E_TRY(nat_launch_pcg_init(e->node_keys, e->d_counts, e->D, nullU, e->type, e->pcg, e->stream));  // codes, r = b
    e->solution_fresh = false;  // pcg.x will hold x_k
    e->warm_ok = false;
    E_TRY(mg_setup_problem(e, true));
    const MgLevel& c = e->mg.L[e->mg.levels - 1];
    const LpGrid G = mg_lp_grid(e, nullptr);
    const int grid = mg_coarse_grid(e);
    if (sample >= 0) {
        // the coarsest right-hand side that one V-cycle makes of the residual
        // after k Jacobi-PCG iterations, and its coarse solution (one-CTA CG)
        for (int k = 0; k < sample; ++k) E_TRY(nat_launch_pcg_iteration(e->node_keys, e->d_counts, e->D, e->pcg, e->stream));
        E_TRY(mg_down(e->mg, nullptr, nat_grid(e, 4), e->stream));
        E_TRY(mg_cg(c, c.r, e->mg_ev, e->mg_s[0], e->mg_s[1], e->mg_s[2], 1e-6, 4000, e->mg_iters, e->stream));
        e->launches += 2u * (uint32_t)sample + (uint32_t)(e->mg.levels - 1) + 1u;
    } else {
        // white noise e on the coarsest fluid cells and r = A e
        E_TRY(lp_noise_sample(G, 0x9E3779B97F4A7C15ull + e->noise_counter++, e->mg_ev, c.r, grid, e->stream));
        e->launches += 2;
    }
    E_TRY(mg_input_scale(e->mg, nullptr, e->stream));
    E_TRY(mg_net_forward(e, G));
    E_CUDA(cudaMemsetAsync(e->lp_scalar, 0, 3 * sizeof(double), e->stream));
    E_TRY(lp_loss_grad(G, e->mg_zn, e->mg_ev, e->mg_wbuf, e->mg_gz, e->lp_scalar, grid, e->stream));
    E_CUDA(cudaMemsetAsync(e->lp.g, 0, sizeof(float) * kLpNumW, e->stream));
    E_TRY(lp_backward_dev(e->lp, G, e->mg.inv_s, e->mg_gz, grid, e->stream));
    e->launches += 1u + 4u + 2u + (e->lp.tensor_cores ? 16u : 14u);
    if (lr > 0.0f) {
        E_TRY(lp_adam(e->lp, lr, e->stream));
        e->launches += 1;
    }
    E_TRY(lp_read_loss(e, loss));
    return lp_check_err(e);
}

extern "C" int flip_get_solve_info(flip_engine* e, flip_solve_info* out) {
    if (!e || !out) return FLIP_ERR_ARG;
    if (e->have_domain) {
        E_CUDA(cudaSetDevice(e->P.device));
        E_TRY(rec_refresh(e));
    }
    *out = e->last_solve;
    return FLIP_OK;
}

extern "C" int flip_set_timing(flip_engine* e, int enable) {
    if (!e) return FLIP_ERR_ARG;
    if (enable && !e->ev[0])
        for (auto& v : e->ev) E_CUDA(cudaEventCreate(&v));
    e->timing = enable != 0;
    return FLIP_OK;
}

extern "C" int flip_get_stage_ms(flip_engine* e, double* ms, int n, int reset) {
    if (!e || !ms || n < 0) return FLIP_ERR_ARG;
    for (int k = 0; k < n && k < FLIP_NUM_STAGES; ++k) ms[k] = e->stage_ms[k];
    if (reset)
        for (double& v : e->stage_ms) v = 0.0;
    return FLIP_OK;
}

extern "C" const char* flip_last_error(flip_engine* e) {
    if (!e) return error_text();
    return e->err.c_str();
}

extern "C" int flip_destroy(flip_engine* e) {
    if (!e) return FLIP_OK;
    cudaSetDevice(e->P.device);
    if (e->up_stream) cudaStreamSynchronize(e->up_stream);
    if (e->down_stream) cudaStreamSynchronize(e->down_stream);
    if (e->stream) cudaStreamSynchronize(e->stream);
    free_arena(e);
    free_ref_voxels(e);
    if (e->solid_tiled) cudaFree(e->solid_tiled);
    if (e->h_small) cudaFreeHost(e->h_small);
    if (e->h_state) cudaFreeHost(e->h_state);
    for (auto& v : e->ev) if (v) cudaEventDestroy(v);
    for (auto& v : e->solve_ev) if (v) cudaEventDestroy(v);
    for (auto& v : e->ev_down) if (v) cudaEventDestroy(v);
    cudaEvent_t evs[3] = {e->ev_start, e->ev_up, e->ev_step};
    for (auto v : evs) if (v) cudaEventDestroy(v);
    if (e->up_stream) cudaStreamDestroy(e->up_stream);
    if (e->down_stream) cudaStreamDestroy(e->down_stream);
    for (auto& c : e->cap_streams) if (c) cudaStreamDestroy(c);
    if (e->lp_warena) cudaFree(e->lp_warena);
    if (e->own_stream && e->stream) cudaStreamDestroy(e->stream);
    delete e;
    return FLIP_OK;
}
