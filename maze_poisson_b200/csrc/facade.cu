// C-ABI facade of libmaze_poisson.so for B200: the symbols, argument meanings and error
// behaviour of the reference's library/src/solver_md.c (plus the enum/string getters of
// grid_general.c, particles.c, integrator_general.c and the serial MPI stubs of
// mpi_base.c), so that maze_poisson/c_api (ctypes) loads it unchanged.
//
// One global system lives on the GPU. Host<->device traffic happens only where the ABI
// moves data: the initialisers and setters (H2D), the getters (D2H) and the scalar
// returns of solver_update_charges / solver_update_field / solver_compute_forces_noel.
// Fatal conditions print a message and exit(1) exactly where the reference does.
#include <cmath>
#include <cstring>
#include <algorithm>
#include <vector>

#include "engine.cuh"
#include "fft.cuh"
#include "mixed.cuh"
#include "particles.cuh"
#include "pb.cuh"
#include "resident.cuh"

namespace mzb {

void fatal_cuda(cudaError_t e, const char* what, const char* file, int line) {
    fprintf(stderr, "maze_poisson_b200: CUDA error '%s' in %s (%s:%d)\n", cudaGetErrorString(e), what,
            file, line);
    exit(1);
}
void fatal(const char* msg) {
    fprintf(stderr, "maze_poisson_b200: %s\n", msg);
    exit(1);
}
unsigned long long g_kernel_launches = 0;

namespace {

enum GridType { G_LCG = 0, G_FFT = 1, G_MG = 2, G_MAZE_LCG = 3, G_MAZE_MG = 4 };
enum Precond { P_NONE = 0, P_JACOBI = 1, P_MG = 2, P_SSOR = 3, P_BLOCKJACOBI = 4 };

const char* kGridNames[5] = {"LCG", "FFT", "MULTIGRID", "MAZE-LCG", "MAZE-MULTIGRID"};
const char* kPrecondNames[5] = {"NONE", "JACOBI", "MG", "SSOR", "BLOCKJACOBI"};
const char* kPotentialNames[3] = {"TF", "LJ", "SC"};
const char* kCasNames[3] = {"CIC", "SPL_QUADR", "SPL_CUBIC"};
const char* kIntegratorNames[2] = {"OVRVO", "VERLET"};

// Host-to-device copies and zero fills that have landed when they return. The blocking
// cudaMemcpy / cudaMemset run on the legacy default stream, which the library's
// non-blocking streams do not wait for, and an upload from pageable memory may return
// before its last DMA completes; waiting on the legacy stream orders them before any
// kernel launched afterwards.
void upload(void* d, const void* h, size_t bytes) {
    if (bytes == 0) return;
    MZB_CHECK(cudaMemcpy(d, h, bytes, cudaMemcpyHostToDevice));
    MZB_CHECK(cudaStreamSynchronize(cudaStreamLegacy));
}
void zero_fill(void* d, size_t bytes) {
    MZB_CHECK(cudaMemset(d, 0, bytes));
    MZB_CHECK(cudaStreamSynchronize(cudaStreamLegacy));
}
void copy_d2d(void* d, const void* src, size_t bytes) {
    MZB_CHECK(cudaMemcpy(d, src, bytes, cudaMemcpyDeviceToDevice));
    MZB_CHECK(cudaStreamSynchronize(cudaStreamLegacy));
}

template <class T>
T* dalloc(size_t count) {
    if (count == 0) count = 1;
    T* p = static_cast<T*>(dev_alloc(sizeof(T) * count));
    zero_fill(p, sizeof(T) * count);
    return p;
}
template <class T>
void dfree(T*& p) {
    dev_free(p);
    p = nullptr;
}

struct GridState {
    bool ready = false;
    int type = 0, precond = 0, n = 0;
    double L = 0, h = 0, tol = 0, eps_s = 1, eps_int = 1;
    long m = 0;
    double* q = nullptr;
    uint32_t* qmask = nullptr;  // spreading's nonzero-charge segments (n % 64 == 0; spread_charges)
    double* buf[3] = {nullptr, nullptr, nullptr};  // phi / phi_prev / spare (renamed)
    int iphi = 0, iprev = 1, ispare = 2;
    double* y = nullptr;
    double *r = nullptr, *p0 = nullptr, *p1 = nullptr, *Ap = nullptr, *v = nullptr, *rf = nullptr,
           *tmp = nullptr;
    double *rc = nullptr, *ec = nullptr, *cr = nullptr, *cp0 = nullptr, *cp1 = nullptr, *cAp = nullptr;
    FftPoisson fft;
    // field-solve form: 0 the reference's FP64 algorithms, 1 mixed precision (FP32
    // multigrid + FP64 refinement), 2 FP64 multigrid (the same V-cycle in FP64)
    int precision = 0;
    double mixed_tol = 0.0;   // > 0 overrides tol for the mixed solve
    int nlev = 0;
    int lev_n[kMixedMaxLevels] = {};
    void* lev_x[kMixedMaxLevels] = {};  // float (precision 1) or double (precision 2)
    void* lev_b[kMixedMaxLevels] = {};
    void* lev_r[kMixedMaxLevels] = {};
    void* lev_g = nullptr;    // Green's function of the coarsest level (direct solve) or null
    int lev_fp64 = 0;         // the levels above hold doubles
    bool coarse_team = false; // the coarsest level (n <= kMixedTeamDirectN) is solved by the whole team
    bool coarse_fft = false;  // the coarsest level (mixed_fft_coarse_ok) is solved by the team by FFT
    void* lev_spec = nullptr; // its half spectrum
    double* lev_hint = nullptr;  // the last solve's first residual max (scale of an FP16 level 0)
    int plan = -1;            // first level that may be solved by FFT (mzb_set_mixed_plan; -1: default)
    // red-black GS sweeps before / after the coarse correction of the multigrid forms
    // (mzb_set_mixed_sweeps): V(3,2) needs one refinement fewer than V(2,2) at tol 1e-8 to
    // 1e-10 on 64^3 to 256^3 grids, for less time in all
    int nu1 = 3, nu2 = 2;
    double batch_cost = 1.0;  // batched-solve time per grid point relative to other sizes (mzb_batch_autotune)
    int lev_plan = -1;        // the plan the current levels were built for
    void* halo = nullptr;      // work area of the resident kernels (ensure_halo)
    double* bj_inv = nullptr;  // block-Jacobi block inverse (1000 x 1000) on BLOCKJACOBI grids
    // Poisson-Boltzmann (solver_initialize_grid_pois_boltz, grid_general.c:84-100)
    bool pb = false;
    PbGrid pbg;

    double* phi() const { return buf[iphi]; }
    double* phi_prev() const { return buf[iprev]; }
};

struct System {
    int device = 0;
    cudaStream_t stream = nullptr;
    GridState G;
    ParticleDev P;
    IntegratorDev I;
    bool parts_ready = false, integ_ready = false;
    double* partials = nullptr;
    GridBarrier* bar = nullptr;
    int* result = nullptr;       // device
    int* result_h = nullptr;     // pinned
    double* red_h = nullptr;     // pinned copy of P.red
    double* scratch_d = nullptr; // small device scratch (energies, reductions)
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;  // around the last solver-engine launch
    float last_solve_ms = 0.f;
    int last_solve_iters = 0;
    double q_tot = 0.0;           // charge of the last spreading; persists like solver_md.c:16
    uint64_t epoch = 0;           // bumped by host-side changes that batched-step graphs bake in
    double* qtot_d = nullptr;     // device copy of q_tot (batched steps check charge on the device)
    std::vector<double> pb_radii; // host copy of the PB solvation radii
    int* err_d = nullptr;         // batched steps: [0] charge error, [2] solve failure
};

System* g = nullptr;             // the selected system
std::vector<System*> g_systems;  // handle -> system (null once destroyed)
int g_current = -1;
bool g_quiet = false;

void touch(System& s) { s.epoch++; }

System& sys() {
    if (!g) fatal("solver_initialize() has not been called");
    return *g;
}
GridState& grid() {
    System& s = sys();
    if (!s.G.ready) fatal("solver_initialize_grid() has not been called");
    return s.G;
}
ParticleDev& parts() {
    System& s = sys();
    if (!s.parts_ready) fatal("solver_initialize_particles() has not been called");
    return s.P;
}

void sync() { MZB_CHECK(cudaStreamSynchronize(sys().stream)); }

void free_grid(GridState& G) {
    dfree(G.q);
    dfree(G.qmask);
    for (auto& b : G.buf) dfree(b);
    dfree(G.y);
    dfree(G.r); dfree(G.p0); dfree(G.p1); dfree(G.Ap); dfree(G.v); dfree(G.rf); dfree(G.tmp);
    dfree(G.rc); dfree(G.ec); dfree(G.cr); dfree(G.cp0); dfree(G.cp1); dfree(G.cAp);
    G.fft.release();
    dfree(G.bj_inv);
    dfree(G.halo);
    dfree(G.pbg.ex); dfree(G.pbg.ey); dfree(G.pbg.ez); dfree(G.pbg.k2); dfree(G.pbg.dg);
    dfree(G.pbg.cex); dfree(G.pbg.cey); dfree(G.pbg.cez); dfree(G.pbg.ck2); dfree(G.pbg.cdg);
    G.pbg = PbGrid{};
    G.pb = false;
    for (int l = 0; l < kMixedMaxLevels; l++) {
        dev_free(G.lev_x[l]);
        dev_free(G.lev_b[l]);
        dev_free(G.lev_r[l]);
        G.lev_x[l] = G.lev_b[l] = G.lev_r[l] = nullptr;
    }
    dev_free(G.lev_g);
    G.lev_g = nullptr;
    dev_free(G.lev_spec);
    G.lev_spec = nullptr;
    dev_free(G.lev_hint);
    G.lev_hint = nullptr;
    G.nlev = 0;
    G.coarse_team = false;
    G.coarse_fft = false;
    G.ready = false;
}

// Mixed precision needs at least three multigrid levels (n, n/2, n/4 even) and the
// plain Laplacian (Poisson-Boltzmann grids stay on the FP64 solvers).
bool mixed_supported(const GridState& G) {
    int sizes[kMixedMaxLevels];
    const int L = mixed_levels(G.n, sizes);
    return G.type != 1 && !G.pb && G.n <= kMixedMaxN && L >= 3 && mixed_small_level(L, sizes) >= 1;
}

void free_mixed_levels(GridState& G) {
    for (int l = 0; l < kMixedMaxLevels; l++) {
        dev_free(G.lev_x[l]);
        dev_free(G.lev_b[l]);
        dev_free(G.lev_r[l]);
        G.lev_x[l] = G.lev_b[l] = G.lev_r[l] = nullptr;
    }
    dev_free(G.lev_g);
    G.lev_g = nullptr;
    dev_free(G.lev_spec);
    G.lev_spec = nullptr;
    dev_free(G.lev_hint);
    G.lev_hint = nullptr;
    G.nlev = 0;
    G.coarse_team = false;
    G.coarse_fft = false;
}

// First level that may be solved by FFT: 1, or from MZB_MIXED_COARSE (a tuning aid) "fft2"
// -> 2, "levels" -> none (the hierarchy down to kMixedTeamDirectN).
int mixed_fft_level() {
    static const int lf = [] {
        const char* e = getenv("MZB_MIXED_COARSE");
        if (e == nullptr) return 1;
        if (strcmp(e, "fft2") == 0) return 2;
        if (strcmp(e, "levels") == 0) return kMixedMaxLevels;
        return 1;
    }();
    return lf;
}

void ensure_mixed_levels(GridState& G) {
    const int fp64 = G.precision == 2 ? 1 : 0;
    const int lf = G.plan >= 0 ? (G.plan == 0 ? kMixedMaxLevels : G.plan) : mixed_fft_level();
    if (G.nlev && (G.lev_fp64 != fp64 || G.lev_plan != lf)) free_mixed_levels(G);  // another form or plan
    if (G.nlev) return;
    G.lev_fp64 = fp64;
    G.lev_plan = lf;
    const size_t w = fp64 ? sizeof(double) : sizeof(float);
    G.nlev = mixed_levels(G.n, G.lev_n);
    G.coarse_team = false;
    G.coarse_fft = false;
    // Stop at the first level the team solves exactly: by FFT when one of the levels from lf
    // on has an FFT size (lf: the grid's plan, else mixed_fft_level(), 1 unless
    // MZB_MIXED_COARSE=fft2 / levels), else by the Green's function at <= kMixedTeamDirectN
    // points per side.
    for (int l = lf; l < G.nlev; l++)
        if (mixed_fft_coarse_ok(G.lev_n[l])) {
            G.nlev = l + 1;
            G.coarse_fft = true;
            break;
        }
    if (!G.coarse_fft)
        for (int l = 1; l < G.nlev; l++)
            if (G.lev_n[l] <= kMixedTeamDirectN) {
                G.nlev = l + 1;
                G.coarse_team = true;
                break;
            }
    for (int l = 0; l < G.nlev; l++) {
        const size_t m = (size_t)G.lev_n[l] * G.lev_n[l] * G.lev_n[l];
        G.lev_x[l] = dev_alloc(m * w);
        G.lev_b[l] = dev_alloc(m * w);
        G.lev_r[l] = dev_alloc(m * w);
        zero_fill(G.lev_x[l], m * w);
    }
    const int nc = G.lev_n[G.nlev - 1];
    if (G.coarse_fft) G.lev_spec = dev_alloc((size_t)nc * nc * (nc / 2 + 1) * 2 * w);
    G.lev_hint = static_cast<double*>(dev_alloc(sizeof(double)));
    zero_fill(G.lev_hint, sizeof(double));
    if (G.coarse_team || (nc <= kMixedDirectN && mixed_small_level(G.nlev, G.lev_n) < G.nlev)) {
        const size_t N = (size_t)nc * nc * nc;
        G.lev_g = dev_alloc(N * w);
        if (fp64) {
            std::vector<double> g(N);
            mixed_coarse_green(nc, g.data());
            upload(G.lev_g, g.data(), N * w);
        } else {
            std::vector<float> g(N);
            mixed_coarse_green(nc, g.data());
            upload(G.lev_g, g.data(), N * w);
        }
    }
}

void free_particles(ParticleDev& P) {
    dfree(P.types); dfree(P.pos); dfree(P.vel); dfree(P.fe); dfree(P.fn); dfree(P.ft);
    dfree(P.mass); dfree(P.chg); dfree(P.tab); dfree(P.base); dfree(P.wgt);
    dfree(P.tile_count); dfree(P.tile_start); dfree(P.tile_fill); dfree(P.tile_ions); dfree(P.tile_part);
    dfree(P.cell_of); dfree(P.cell_count); dfree(P.cell_start); dfree(P.cell_fill);
    dfree(P.cell_ions); dfree(P.srank); dfree(P.spos); dfree(P.stype); dfree(P.fpart);
    dfree(P.epart); dfree(P.red); dfree(P.flags); dfree(P.partial);
    dfree(P.tf_st); dfree(P.tf_gstart); dfree(P.tf_gent); dfree(P.tf_box);
    dfree(P.radii); dfree(P.fdb); dfree(P.fib); dfree(P.fnp); dfree(P.pb_part);
    P = ParticleDev{};
}

// Linked cells that order the ions for the pair-force kernel: about 16 ions per cell, at
// least one cell per side.
// r^2 beyond which the Born-Mayer terms of a Tosi-Fumi pair, A B exp(B (sigma - r)) in
// the force and A exp(B (sigma - r)) in the energy, are both below 1e-21 hartree (/bohr),
// so the pair-force kernel leaves the exponential out beyond it. Summed over all of an
// ion's partners (N = 16000: < 2e-17 hartree/bohr) that stays below the rounding of the
// ion's force sum (~1e-16 for forces of 1e-2 over thousands of pairs); for NaCl it is
// r ~ 31 bohr of r_cut = 78 at N = 16000.
double tf_exp_r2_limit(double A, double B, double sg) {
    const double m = std::max(fabs(A * B), fabs(A));
    if (m == 0.0) return 0.0;
    if (!(B > 0.0)) return INFINITY;
    const double r = sg - log(1e-21 / m) / B;
    return r > 0.0 ? r * r : 0.0;
}

void set_cells(ParticleDev& P, int nc) {
    dfree(P.cell_count); dfree(P.cell_start); dfree(P.cell_fill);
    P.nc = nc < 1 ? 1 : nc;
    P.ncell = P.nc * P.nc * P.nc;
    P.cell_count = dalloc<int32_t>(P.ncell);
    P.cell_start = dalloc<int32_t>(P.ncell + 1);
    P.cell_fill = dalloc<int32_t>(P.ncell);
}

// A device copy of the block-Jacobi block inverse (the caller frees it).
double* device_block_inverse() {
    const std::vector<double>& inv = block_jacobi_inverse();
    double* d = dalloc<double>(inv.size());
    upload(d, inv.data(), sizeof(double) * inv.size());
    return d;
}

// Point the engine's PB operator at the coefficients of g.
void set_pb_operator(EngineArgs& a, const PbGrid& g) {
    a.pb = 1;
    a.ex = g.ex; a.ey = g.ey; a.ez = g.ez; a.dg = g.dg;
    a.cex = g.cex; a.cey = g.cey; a.cez = g.cez; a.cdg = g.cdg;
}

// The resident kernels' work area, allocated at the first solve that can use it.
void ensure_halo(GridState& G) {
    if (G.halo) return;
    const size_t bytes = resident_halo_bytes(G.n);
    if (bytes) G.halo = dalloc<unsigned char>(bytes);
}

EngineArgs engine_base(System& s) {
    GridState& G = s.G;
    ensure_halo(G);
    EngineArgs a{};
    a.n = G.n;
    a.tol = G.tol;
    a.halo = G.halo;
    a.r = G.r; a.p0 = G.p0; a.p1 = G.p1; a.Ap = G.Ap; a.v = G.v; a.rf = G.rf; a.tmp = G.tmp;
    a.rc = G.rc; a.ec = G.ec; a.cr = G.cr; a.cp0 = G.cp0; a.cp1 = G.cp1; a.cAp = G.cAp;
    a.partials = s.partials;
    a.bar = s.bar;
    a.result = s.result;
    a.q = G.q;
    a.y = G.y;
    a.bj_inv = G.bj_inv;
    if (G.pb) set_pb_operator(a, G.pbg);
    return a;
}

// Launch the solver for `a`: the resident kernels where size and program allow, then the
// TMA-staged CG, then the general engine (MZB_ENGINE=generic: always that).
void launch_solver(const EngineArgs& a, cudaStream_t stream) {
    static const bool generic_only = getenv("MZB_ENGINE") && strcmp(getenv("MZB_ENGINE"), "generic") == 0;
    if (!generic_only && (resident_cg_launch(a, stream) || resident_mg_launch(a, stream) || cg_fast_launch(a, stream))) return;
    engine_launch(a, stream);
}

// Run the engine and return its result; an engine failure (a barrier that timed out)
// is reported and turned into -1 ("not converged").
int run_engine(System& s, const EngineArgs& a) {
    MZB_CHECK(cudaEventRecord(s.ev0, s.stream));
    // MZB_PHASE_TIMING=1: time-stamp the phases of the CG kernels and print them (debug aid)
    static const bool stamps_on = getenv("MZB_PHASE_TIMING") != nullptr;
    static unsigned long long* stamps_d = nullptr;
    EngineArgs b = a;
    if (stamps_on) {
        if (!stamps_d) MZB_CHECK(cudaMalloc(&stamps_d, sizeof(unsigned long long) * 96));
        MZB_CHECK(cudaMemsetAsync(stamps_d, 0, sizeof(unsigned long long) * 96, s.stream));
        b.stamps = stamps_d;
    }
    launch_solver(b, s.stream);
    if (stamps_on) {
        unsigned long long h[96];
        MZB_CHECK(cudaMemcpyAsync(h, stamps_d, sizeof(h), cudaMemcpyDeviceToHost, s.stream));
        MZB_CHECK(cudaStreamSynchronize(s.stream));
        if (h[0]) {
            fprintf(stderr, "[cg phases us] pre %.2f sync %.2f init %.2f |", (h[1] - h[0]) * 1e-3,
                    (h[2] - h[1]) * 1e-3, 0.0);
            for (int it = 0; it + 1 < kCgStampIters; it++) {
                const unsigned long long* t = h + 4 + 4 * it;
                if (!t[0] || !t[4]) break;
                fprintf(stderr, " A %.2f redA %.2f B %.2f redB %.2f |", (t[0] - (it ? t[-1] : h[2])) * 1e-3,
                        (t[1] - t[0]) * 1e-3, (t[2] - t[1]) * 1e-3, (t[3] - t[2]) * 1e-3);
            }
            if (h[40]) fprintf(stderr, "\n[cg phase A slabs us: sync+issue, p_new, stencil]");  // cg_fast only
            for (int e = 0; e < 18 && h[40 + 3 * e]; e++) {
                const unsigned long long prev = e ? h[39 + 3 * e] : h[2];
                fprintf(stderr, " %.2f,%.2f,%.2f", (h[40 + 3 * e] - prev) * 1e-3, (h[41 + 3 * e] - h[40 + 3 * e]) * 1e-3,
                        (h[42 + 3 * e] - h[41 + 3 * e]) * 1e-3);
            }
            fprintf(stderr, "\n");
        }
    }
    MZB_CHECK(cudaEventRecord(s.ev1, s.stream));
    MZB_CHECK(cudaMemcpyAsync(s.result_h, s.result, 2 * sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    MZB_CHECK(cudaStreamSynchronize(s.stream));
    MZB_CHECK(cudaEventElapsedTime(&s.last_solve_ms, s.ev0, s.ev1));
    s.last_solve_iters = s.result_h[0];
    if (s.result_h[1] != 0) {
        fprintf(stderr, "maze_poisson_b200: solver engine aborted (grid barrier timeout)\n");
        return -1;
    }
    return s.result_h[0];
}

// Mixed-precision solve of program `prog` (see mixed.cu); returns refinement steps or -1.
// Arguments of the mixed-precision solve of program `prog` for system s (writes the new
// field into the spare buffer; the caller rotates the buffers afterwards).
MixedArgs mixed_args(System& s, int prog, double cst) {
    GridState& G = s.G;
    ensure_mixed_levels(G);
    MixedArgs m{};
    m.prog = prog;
    m.n = G.n;
    m.tol = G.mixed_tol > 0 ? G.mixed_tol : G.tol;
    m.c = cst;
    m.max_outer = 100;
    m.nu1 = G.nu1;
    m.nu2 = G.nu2;
    m.coarse_sweeps = 16;
    m.nlev = G.nlev;
    m.lsmall = G.coarse_team || G.coarse_fft ? G.nlev : mixed_small_level(G.nlev, G.lev_n);
    m.coarse_g = G.lev_g;
    m.coarse_fft = G.coarse_fft ? 1 : 0;

    m.coarse_spec = G.lev_spec;
    m.fp64 = G.lev_fp64;
    // FP16 storage of level 0 at 256^3, where the level-0 passes stream from HBM (at 128^3
    // they run from L2 and FP16 measured slower). The correction only has to cut the
    // residual by the V-cycle's factor each refinement; the FP64 residual and update keep
    // the solution's accuracy. The batched solve keeps FP32 (mixed_batch_kernel).
    m.level0_fp16 = !m.fp64 && G.n == 256 ? 1 : 0;
    m.scale_hint = G.lev_hint;
    m.coarse_team = G.coarse_team ? 1 : 0;
    for (int l = 0; l < G.nlev; l++) {
        m.lev_n[l] = G.lev_n[l];
        m.lev_x[l] = G.lev_x[l];
        m.lev_b[l] = G.lev_b[l];
        m.lev_r[l] = G.lev_r[l];
    }
    m.q = G.q;
    m.qmask = G.qmask;
    m.phi_old = G.phi();
    m.phi_prev = G.phi_prev();
    m.phi_new = G.buf[G.ispare];
    m.y = G.y;
    m.tmp = G.tmp;
    m.partials = s.partials;
    m.bar = s.bar;
    m.result = s.result;
    return m;
}

// The mixed-precision program of an MD-step field update for the grid's method and its
// right-hand-side constant (the mixed branch of solver_update_field).
int mixed_update_prog(const GridState& G, double& cst) {
    if (G.type == G_LCG || G.type == G_MG) {
        cst = -4 * kPi / G.h / G.eps_s;
        return G.type == G_LCG ? PROG_LCG_UPDATE : PROG_MG_UPDATE;
    }
    cst = (4 * kPi) / (G.h * G.eps_s);
    return G.type == G_MAZE_LCG ? PROG_MAZE_LCG : PROG_MAZE_MG;
}

int run_mixed(System& s, int prog, double cst) {
    GridState& G = s.G;
    MixedArgs m = mixed_args(s, prog, cst);
    // MZB_PHASE_TIMING=1: time-stamp the phases of each refinement step and print them
    static const bool stamps_on = getenv("MZB_PHASE_TIMING") != nullptr;
    static unsigned long long* stamps_d = nullptr;
    if (stamps_on) {
        if (!stamps_d) MZB_CHECK(cudaMalloc(&stamps_d, sizeof(unsigned long long) * kMixedStampSlots));
        MZB_CHECK(cudaMemsetAsync(stamps_d, 0, sizeof(unsigned long long) * kMixedStampSlots, s.stream));
        m.stamps = stamps_d;
    }
    MZB_CHECK(cudaEventRecord(s.ev0, s.stream));
    mixed_launch(m, s.stream);
    MZB_CHECK(cudaEventRecord(s.ev1, s.stream));
    if (stamps_on) {
        unsigned long long h[kMixedStampSlots];
        MZB_CHECK(cudaMemcpyAsync(h, stamps_d, sizeof(h), cudaMemcpyDeviceToHost, s.stream));
        MZB_CHECK(cudaStreamSynchronize(s.stream));
        fprintf(stderr, "[mixed phases us] setup %.2f |", (h[1] - h[0]) * 1e-3);
        for (int o = 0; o < 8; o++) {
            const unsigned long long* t = h + 2 + 8 * o;
            if (!t[0] || !t[1]) break;
            double rmax;
            memcpy(&rmax, &t[7], sizeof(double));
            fprintf(stderr, " r=%.2e resid %.2f", rmax, (t[1] - t[0]) * 1e-3);
            if (!t[6]) break;
            fprintf(stderr, " down %.2f small %.2f up %.2f esum %.2f upd %.2f |", (t[2] - t[1]) * 1e-3,
                    (t[3] - t[2]) * 1e-3, (t[4] - t[3]) * 1e-3, (t[5] - t[4]) * 1e-3, (t[6] - t[5]) * 1e-3);
        }
        const unsigned long long* f = h + 2 + 8 * 8;
        if (f[0] && f[7]) {
            fprintf(stderr, "[coarse FFT us, refinement 1] twiddles %.2f planes-i %.2f sync %.2f planes-kj %.2f sync %.2f planes-i %.2f sync %.2f",
                    (f[1] - f[0]) * 1e-3, (f[2] - f[1]) * 1e-3, (f[3] - f[2]) * 1e-3, (f[4] - f[3]) * 1e-3,
                    (f[5] - f[4]) * 1e-3, (f[6] - f[5]) * 1e-3, (f[7] - f[6]) * 1e-3);
        }
        fprintf(stderr, "\n");
    }
    MZB_CHECK(cudaMemcpyAsync(s.result_h, s.result, 2 * sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    MZB_CHECK(cudaStreamSynchronize(s.stream));
    MZB_CHECK(cudaEventElapsedTime(&s.last_solve_ms, s.ev0, s.ev1));
    s.last_solve_iters = s.result_h[0];
    if (s.result_h[1] != 0) {
        fprintf(stderr, "maze_poisson_b200: mixed solver aborted (grid barrier timeout)\n");
        return -1;
    }
    // phi_prev <- old phi, phi <- new
    const int old = G.iphi;
    G.iphi = G.ispare;
    G.ispare = G.iprev;
    G.iprev = old;
    return s.result_h[0];
}

// FFT Poisson solve of the current charge grid into phi (in place; FFT grids keep no
// previous field), timed like the iterative solves.
void run_fft(System& s) {
    GridState& G = s.G;
    MZB_CHECK(cudaEventRecord(s.ev0, s.stream));
    G.fft.solve(G.q, G.phi(), s.stream);
    MZB_CHECK(cudaEventRecord(s.ev1, s.stream));
    MZB_CHECK(cudaStreamSynchronize(s.stream));
    MZB_CHECK(cudaEventElapsedTime(&s.last_solve_ms, s.ev0, s.ev1));
    s.last_solve_iters = 0;
}

void require_mg_size(int n) {
    // multigrid.c:114-121: at least one level of recursion, n/2 >= 16
    if (n / 2 < 16 || n % 2) fatal("Multigrid: requires an even grid with n/2 >= 16");
}

// -4 pi / h, divided by eps_s unless the PB operator carries the dielectric
// (grid_lcg.c:100-110)
double rhs_const(const GridState& G) {
    double c = -4 * kPi / G.h;
    if (!G.pb) c /= G.eps_s;
    return c;
}

// (4 pi) / h of the MaZe constraint: h <- h * eps_s on Poisson grids (grid_maze_lcg.c:158,
// grid_maze_multigrid.c:133), plain h with PB (verlet.c:178, 232)
double maze_const(const GridState& G) { return G.pb ? (4 * kPi) / G.h : (4 * kPi) / (G.h * G.eps_s); }

// Check the PB boxes fit the grid and size the force partials (the reference writes out of
// bounds when a box of +-(floor((r_s+w)/h)+2) points is wider than the grid).
void ensure_pb_forces(System& s) {
    GridState& G = s.G;
    ParticleDev& P = s.P;
    if (P.pb_range > 0) return;
    int rmax = 0;
    for (double r : s.pb_radii) {
        const int rg = (int)floor((r + G.pbg.w) / G.h) + 2;
        rmax = rg > rmax ? rg : rmax;
    }
    if (rmax >= G.n) fatal("Poisson-Boltzmann: an ion's solvation box is wider than the grid");
    P.pb_range = rmax;
    P.pb_part = dalloc<double>((size_t)P.np * (2 * rmax + 1) * 9);
}

}  // namespace
}  // namespace mzb

using namespace mzb;

extern "C" {

// ---------------------------------------------------------------- serial MPI stubs
int init_mpi(void) { return 0; }  // mpi_base.c:169-177 (serial build)
int get_rank(void) { return 0; }

// ---------------------------------------------------------------- enum tables
int get_grid_type_num(void) { return 5; }
char* get_grid_type_str(int i) { return (char*)kGridNames[i]; }
int get_precond_type_num(void) { return 5; }
char* get_precond_type_str(int i) { return (char*)kPrecondNames[i]; }
int get_potential_type_num(void) { return 3; }
char* get_potential_type_str(int i) { return (char*)kPotentialNames[i]; }
int get_ca_scheme_type_num(void) { return 3; }
char* get_ca_scheme_type_str(int i) { return (char*)kCasNames[i]; }
int get_integrator_type_num(void) { return 2; }
char* get_integrator_type_str(int i) { return (char*)kIntegratorNames[i]; }

// ---------------------------------------------------------------- lifecycle
void solver_initialize(void) {
    if (!g) {
        g = new System();
        g_systems.push_back(g);
        g_current = (int)g_systems.size() - 1;
    }
    const char* dev = getenv("MZB_DEVICE");
    g->device = dev ? atoi(dev) : 0;
    g_quiet = getenv("MZB_QUIET") != nullptr;
    MZB_CHECK(cudaSetDevice(g->device));
    if (!g->stream) MZB_CHECK(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    if (!g->partials) {
        const int blocks = engine_grid_blocks();
        g->partials = dalloc<double>((size_t)2 * 8 * blocks);
        g->bar = dalloc<GridBarrier>(1);
        g->result = dalloc<int>(2);
        MZB_CHECK(cudaMallocHost(&g->result_h, 2 * sizeof(int)));
        MZB_CHECK(cudaMallocHost(&g->red_h, 8 * sizeof(double)));
        g->scratch_d = dalloc<double>(4096);
        MZB_CHECK(cudaEventCreate(&g->ev0));
        MZB_CHECK(cudaEventCreate(&g->ev1));
    }
    if (!g_quiet) {
        cudaDeviceProp prop;
        MZB_CHECK(cudaGetDeviceProperties(&prop, g->device));
        printf("******************************************************\n");
        printf("* MAZE_POISSON (B200 CUDA build)\n");
        printf("*   GPU     %s, %d SMs\n", prop.name, prop.multiProcessorCount);
        printf("******************************************************\n");
    }
}

void solver_initialize_grid(int n, double L, double h, double tol, double eps, double eps_int,
                            int grid_type, int precond_type) {
    System& s = sys();
    GridState& G = s.G;
    touch(s);
    if (G.ready) free_grid(G);
    if (grid_type < 0 || grid_type > 4) fatal("invalid grid type");
    if (n < 2) fatal("grid size must be at least 2");
    G.type = grid_type;
    G.precond = precond_type;
    G.n = n;
    G.L = L;
    G.h = h;
    G.tol = tol;
    G.eps_s = eps;
    G.eps_int = eps_int;
    G.m = (long)n * n * n;
    G.iphi = 0; G.iprev = 1; G.ispare = 2;
    {
        const char* pm = getenv("MZB_PRECISION");
        G.precision = (pm && strcmp(pm, "mixed") == 0) ? 1 : (pm && strcmp(pm, "fp64mg") == 0) ? 2 : 0;
    }
    G.q = dalloc<double>(G.m);
    if (n % 64 == 0) G.qmask = dalloc<uint32_t>(((size_t)G.m / 64 + 31) / 32);
    G.buf[0] = dalloc<double>(G.m);
    if (grid_type == G_FFT) {
        G.fft.init(n, L, h);
    } else {
        if (grid_type == G_MG || grid_type == G_MAZE_MG) require_mg_size(n);
        if (n % 2) fatal("this build requires an even grid size (red-black smoothing, multigrid)");
        G.buf[1] = dalloc<double>(G.m);
        G.buf[2] = dalloc<double>(G.m);
        G.y = dalloc<double>(G.m);
        G.r = dalloc<double>(G.m); G.p0 = dalloc<double>(G.m); G.p1 = dalloc<double>(G.m);
        G.Ap = dalloc<double>(G.m); G.tmp = dalloc<double>(G.m);
        const bool mg = grid_type == G_MG || grid_type == G_MAZE_MG ||
                        (grid_type == G_MAZE_LCG && precond_type == P_MG);
        if (mg) {
            require_mg_size(n);
            const long mc = G.m / 8;
            G.v = dalloc<double>(G.m); G.rf = dalloc<double>(G.m);
            G.rc = dalloc<double>(mc); G.ec = dalloc<double>(mc); G.cr = dalloc<double>(mc);
            G.cp0 = dalloc<double>(mc); G.cp1 = dalloc<double>(mc); G.cAp = dalloc<double>(mc);
        }
        if (grid_type == G_MAZE_LCG && (precond_type == P_SSOR || precond_type == P_BLOCKJACOBI))
            G.v = dalloc<double>(G.m);  // v = M^-1 r
        if ((grid_type == G_LCG || grid_type == G_MAZE_LCG) && precond_type == P_BLOCKJACOBI)
            G.bj_inv = device_block_inverse();  // precond_blockjacobi_init (grid_lcg.c:75-78)
    }
    G.ready = true;
}

// grid_pb_init (grid_general.c:84-100): face coefficients, screening term and the PB
// operator's diagonal on the grid (and the coarse grid of the PB V-cycle on MULTIGRID and
// MAZE-MULTIGRID grids); filled by solver_update_eps_k2.
void solver_initialize_grid_pois_boltz(double w, double kbar2, int nonpolar_enabled) {
    System& s = sys();
    GridState& G = grid();
    touch(s);
    PbGrid& g = G.pbg;
    if (!G.pb) {
        g.ex = dalloc<double>(G.m); g.ey = dalloc<double>(G.m); g.ez = dalloc<double>(G.m);
        g.k2 = dalloc<double>(G.m); g.dg = dalloc<double>(G.m);
        if (G.type == G_MG || G.type == G_MAZE_MG) {
            const long mc = G.m / 8;
            g.cex = dalloc<double>(mc); g.cey = dalloc<double>(mc); g.cez = dalloc<double>(mc);
            g.ck2 = dalloc<double>(mc); g.cdg = dalloc<double>(mc);
        }
    }
    G.pb = true;
    g.n = G.n;
    g.h = G.h;
    g.w = w;
    g.eps_s = G.eps_s;
    g.eps_int = G.eps_int;
    g.kbar2 = kbar2;
    g.nonpolar = nonpolar_enabled;
    if (s.parts_ready) {  // the force boxes depend on w
        dfree(s.P.pb_part);
        s.P.pb_range = 0;
    }
}

void solver_initialize_particles(int n, int n_typ, double L, double h, int n_p, int pot_type, int cas_type,
                                 int* types, double* pos, double* vel, double* mass, double* charges,
                                 double* pot_params) {
    System& s = sys();
    touch(s);
    if (pot_type < 0 || pot_type > 2) fatal("invalid potential type");
    if (cas_type < 0 || cas_type > 2) fatal("invalid charge assignment scheme");
    if (cas_type != CAS_CIC && n < 4)  // offsets -1..2 would wrap onto the same point
        fatal("B-spline charge assignment needs a grid of at least 4 points per side");
    if (n_typ < 1 || n_typ > 8) fatal("between 1 and 8 particle types are supported");
    if (s.parts_ready) free_particles(s.P);
    s.pb_radii.clear();
    ParticleDev& P = s.P;
    P.cas = cas_type;
    P.np = n_p;
    P.ntyp = n_typ;
    P.n = n;
    P.L = L;
    P.h = h;
    P.rcut = L / 2.0;  // particles.c:189
    const size_t v3 = (size_t)3 * n_p;
    P.types = dalloc<int32_t>(n_p);
    P.pos = dalloc<double>(v3);
    P.vel = dalloc<double>(v3);
    P.fe = dalloc<double>(v3);
    P.fn = dalloc<double>(v3);
    P.ft = dalloc<double>(v3);
    P.mass = dalloc<double>(n_p);
    P.chg = dalloc<double>(n_p);
    P.base = dalloc<int32_t>(v3);
    if (cas_type != CAS_CIC) P.wgt = dalloc<double>((size_t)12 * n_p);
    if (n_p > 0) {
        upload(P.types, types, sizeof(int32_t) * n_p);
        upload(P.pos, pos, sizeof(double) * v3);
        upload(P.vel, vel, sizeof(double) * v3);
        upload(P.mass, mass, sizeof(double) * n_p);
        upload(P.chg, charges, sizeof(double) * n_p);
    }
    // pair-potential constants per type pair, kPairConsts doubles each, with the
    // shifted-force constants at r_cut = L/2
    P.pot = pot_type;
    std::vector<double> tab((size_t)n_typ * n_typ * kPairConsts, 0.0);
    const double rc = L / 2.0, rc6 = pow(rc, 6), rc7 = rc6 * rc, rc8 = rc7 * rc, rc9 = rc8 * rc;
    for (int t = 0; t < n_typ * n_typ; t++) {
        double* o = &tab[kPairConsts * t];
        if (pot_type == POT_TF) {  // particles.c:181-228: [A, B, C, D, sigma, alpha, beta]
            const double A = pot_params[5 * t], B = pot_params[5 * t + 1], C = pot_params[5 * t + 2],
                         D = pot_params[5 * t + 3], sg = pot_params[5 * t + 4];
            const double ea = exp(B * (sg - rc));
            const double vs = A * ea - C / rc6 - D / rc8;
            const double al = A * B * ea - 6 * C / rc7 - 8 * D / rc9;
            const double be = -vs - al * rc;
            o[0] = A; o[1] = B; o[2] = C; o[3] = D; o[4] = sg; o[5] = al; o[6] = be;
            o[7] = tf_exp_r2_limit(A, B, sg);
        } else if (pot_type == POT_LJ) {
            // particles.c:230-266: [sigma, epsilon, alpha, beta]. pot_params holds [sigma,
            // epsilon] per type pair as solver.py:241-270 passes it; the reference reads
            // it with a stride of 4 (particles.c:241), past the array for two or more
            // types -- with one type both agree.
            const double sg = pot_params[2 * t], ep = pot_params[2 * t + 1];
            const double vs = 4 * ep * (pow(sg / rc, 12) - pow(sg / rc, 6));
            const double al = 4 * (12 * ep * pow(sg / rc, 12) - 6 * ep * pow(sg / rc, 6)) / rc;
            o[0] = sg; o[1] = ep; o[2] = al; o[3] = -vs - al * rc;
        } else {  // particles.c:268-295: [nu, d, B, alpha, beta], shared by every pair
            const double nu = pot_params[0], d = pot_params[1], B = pot_params[2];
            const double drp = pow(d / rc, nu);
            const double al = B * nu * drp / rc;
            o[0] = nu; o[1] = d; o[2] = B; o[3] = al; o[4] = -B * drp - al * rc;
        }
    }
    P.tab = dalloc<double>(tab.size());
    upload(P.tab, tab.data(), sizeof(double) * tab.size());
    // spreading tiles over the grid
    P.nti = (n + kTileI - 1) / kTileI;
    P.ntj = (n + kTileJ - 1) / kTileJ;
    P.ntk = (n + kTileK - 1) / kTileK;
    P.ntiles = P.nti * P.ntj * P.ntk;
    P.tile_count = dalloc<int32_t>(P.ntiles);
    P.tile_start = dalloc<int32_t>(P.ntiles + 1);
    P.tile_fill = dalloc<int32_t>(P.ntiles);
    P.tile_part = dalloc<int32_t>((P.ntiles + 1023) / 1024);
    P.tile_ions = dalloc<int32_t>(n_p);
    // linked cells
    P.cell_of = dalloc<int32_t>(n_p);
    P.cell_ions = dalloc<int32_t>(n_p);
    P.srank = dalloc<int32_t>(n_p);
    P.spos = dalloc<double>(v3);
    P.stype = dalloc<int32_t>(n_p);
    const int nc = (int)std::lround(std::cbrt(n_p / 16.0));
    set_cells(P, nc < 1 ? 1 : nc);
    tf_plan(P);
    P.red = dalloc<double>(16);
    P.flags = dalloc<int>(4);
    P.partial = dalloc<double>((size_t)4 * ((n_p + 127) / 128) + 64);
    s.parts_ready = true;
}

// particles_pb_init (particles.c:111-127): solvation radii and the three PB force arrays.
void solver_initialize_particles_pois_boltz(double gamma_np, double beta_np, double* solv_radii) {
    System& s = sys();
    ParticleDev& P = parts();
    touch(s);
    P.gamma_np = gamma_np;
    P.beta_np = beta_np;
    if (!P.fdb) {
        P.radii = dalloc<double>(P.np);
        P.fdb = dalloc<double>((size_t)3 * P.np);
        P.fib = dalloc<double>((size_t)3 * P.np);
        P.fnp = dalloc<double>((size_t)3 * P.np);
    }
    if (P.np > 0) upload(P.radii, solv_radii, sizeof(double) * P.np);
    s.pb_radii.assign(solv_radii, solv_radii + P.np);
    dfree(P.pb_part);
    P.pb_range = 0;
}

void solver_initialize_integrator(int n_p, double dt, double T, double gamma, int itg_type, int itg_enabled) {
    System& s = sys();
    touch(s);
    (void)n_p;
    IntegratorDev& I = s.I;
    const uint64_t seed = I.seed;
    I = IntegratorDev{};
    I.seed = seed;
    I.type = itg_type;
    I.dt = dt;
    if (itg_enabled == 1) {  // *_integrator_init_thermostat
        I.T = T;
        I.enabled = 1;
        if (itg_type == 0) {
            I.c1 = exp(-gamma * dt);
            I.c2 = sqrt(2 / (gamma * dt) * tanh(0.5 * gamma * dt));
        }
    }
    s.integ_ready = true;
}

// solver_md.c:91-107
int solver_update_charges(void) {
    System& s = sys();
    GridState& G = grid();
    ParticleDev& P = parts();
    spread_charges(P, G.q, G.qmask, G.n, G.h, s.stream);
    MZB_CHECK(cudaMemcpyAsync(s.red_h, P.red, sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    sync();
    const double q_loc = s.red_h[0];
    int res = 0;
    if (fabs(s.q_tot - q_loc) > 1e-6) {
        res = 1;
        printf("Charge conservation error: q_tot = %.6f, q_tot_loc = %.6f\n", s.q_tot, q_loc);
        exit(1);
    }
    s.q_tot = q_loc;
    return res;
}

void solver_init_field(void) {
    System& s = sys();
    GridState& G = grid();
    if (G.type == G_FFT) {  // grid_fft.c:135-137
        run_fft(s);
        return;
    }
    if (G.precision >= 1 && mixed_supported(G)) {
        run_mixed(s, PROG_INIT_FIELD, rhs_const(G));
        return;
    }
    EngineArgs a = engine_base(s);
    a.prog = PROG_INIT_FIELD;
    a.c = rhs_const(G);
    a.phi_old = G.phi();
    a.phi_prev = G.phi_prev();
    a.phi_new = G.buf[G.ispare];
    run_engine(s, a);
    // phi_prev <- old phi, phi <- solution
    const int old = G.iphi;
    G.iphi = G.ispare;
    G.ispare = G.iprev;
    G.iprev = old;
}

}  // extern "C"

namespace mzb {
namespace {
int md_steps_deferred(System& s, int n_steps);

// Engine arguments of an MD-step field update on an FP64 grid (the engine branch of
// solver_update_field): the new field goes into the spare buffer.
EngineArgs update_engine_args(System& s) {
    GridState& G = s.G;
    EngineArgs a = engine_base(s);
    a.phi_old = G.phi();
    a.phi_prev = G.phi_prev();
    a.phi_new = G.buf[G.ispare];
    switch (G.type) {
    case G_LCG:
        a.prog = PROG_LCG_UPDATE;
        a.c = rhs_const(G);
        break;
    case G_MAZE_LCG:
        a.prog = PROG_MAZE_LCG;
        a.c = maze_const(G);  // verlet.c:55 with h <- h*eps (grid_maze_lcg.c:158); PB verlet.c:178
        if (G.precond == P_NONE || G.pb) a.precond = PC_IMPLICIT;  // PB ignores it (grid_maze_lcg.c:150-156)
        else if (G.precond == P_JACOBI) a.precond = PC_JACOBI;
        else if (G.precond == P_MG) a.precond = PC_MG;
        else if (G.precond == P_SSOR) a.precond = PC_SSOR;
        else {  // precond_blockjacobi.c:192-197
            if (G.n % kBlockJacobiB) {
                fprintf(stderr, "Error: The size of the input vector is not a multiple of the block size (%d)\n",
                        kBlockJacobiB3);
                fprintf(stderr, "Padding is not implemented yet\n");
                exit(1);
            }
            a.precond = PC_BLOCKJACOBI;
        }
        break;
    case G_MG:
        a.prog = PROG_MG_UPDATE;
        a.c = rhs_const(G);
        break;
    case G_MAZE_MG:
        a.prog = PROG_MAZE_MG;
        a.c = maze_const(G);
        break;
    }
    return a;
}
}  // namespace
}  // namespace mzb

extern "C" {

int solver_update_field(void) {
    System& s = sys();
    GridState& G = grid();
    if (G.type == G_FFT) {  // grid_fft.c:139-143
        run_fft(s);
        return 0;
    }
    if (G.precision >= 1 && mixed_supported(G)) {
        if (G.type == G_MAZE_MG && G.precond != P_NONE) {  // grid_maze_multigrid.c:138-141
            fprintf(stderr, "Maze Multigrid with preconditioner not implemented yet.\n");
            exit(1);
        }
        if (G.type == G_LCG) return run_mixed(s, PROG_LCG_UPDATE, rhs_const(G));
        if (G.type == G_MG) return run_mixed(s, PROG_MG_UPDATE, rhs_const(G));
        return run_mixed(s, G.type == G_MAZE_LCG ? PROG_MAZE_LCG : PROG_MAZE_MG, maze_const(G));
    }
    EngineArgs a = update_engine_args(s);
    const int res = run_engine(s, a);
    const int old = G.iphi;
    G.iphi = G.ispare;
    G.ispare = G.iprev;
    G.iprev = old;
    if (G.type == G_MAZE_MG) {
        if (res == -1) fprintf(stderr, "Warning: Multigrid did not converge after 1000 iterations.\n");
        if (G.precond != P_NONE) {  // grid_maze_multigrid.c:138-141
            fprintf(stderr, "Maze Multigrid with preconditioner not implemented yet.\n");
            exit(1);
        }
    }
    return res;
}

void solver_set_field(double* phi) {
    System& s = sys();
    GridState& G = grid();
    MZB_CHECK(cudaMemcpyAsync(G.phi(), phi, sizeof(double) * G.m, cudaMemcpyHostToDevice, s.stream));
    sync();
}

void solver_set_field_prev(double* phi) {
    System& s = sys();
    GridState& G = grid();
    if (G.type == G_FFT) return;  // no phi_prev (solver_md.c:119-129)
    MZB_CHECK(cudaMemcpyAsync(G.phi_prev(), phi, sizeof(double) * G.m, cudaMemcpyHostToDevice, s.stream));
    sync();
}

// grid_update_eps_and_k2 (grid_general.c:138-301) from the current positions.
void solver_update_eps_k2(void) {
    System& s = sys();
    GridState& G = grid();
    ParticleDev& P = parts();
    if (!G.pb || !P.fdb)
        fatal("solver_update_eps_k2: Poisson-Boltzmann is not initialised for the grid and the particles");
    ensure_pb_forces(s);
    pb_update_coefficients(G.pbg, P.pos, P.radii, P.np, s.stream);
}

void solver_compute_forces_elec(void) {
    System& s = sys();
    GridState& G = grid();
    field_forces(parts(), G.phi(), G.n, G.h, s.stream);
}

double solver_compute_forces_noel(void) {
    System& s = sys();
    ParticleDev& P = parts();
    build_cells(P, s.stream);
    tf_forces(P, s.stream);
    MZB_CHECK(cudaMemcpyAsync(s.red_h + 1, P.red + 1, sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    sync();
    return s.red_h[1];
}

// particles_compute_forces_pb (particles.c:420-775); returns the non-polar energy, which
// the reference never accumulates (always 0).
double solver_compute_forces_pb(void) {
    System& s = sys();
    GridState& G = grid();
    ParticleDev& P = parts();
    if (!G.pb) {
        fprintf(stderr, "Poisson-Boltzmann forces are not enabled in the grid.\n");
        exit(1);
    }
    if (!P.fdb) fatal("solver_compute_forces_pb: solver_initialize_particles_pois_boltz() has not been called");
    ensure_pb_forces(s);
    const double cdb = G.h / (8.0 * kPi);
    const double cnp = -P.gamma_np * G.h / (G.eps_s - G.eps_int);
    pb_forces(G.pbg, G.phi(), P.pos, P.radii, P.np, P.pb_range, cdb, cnp, P.pb_part, P.fdb, P.fib, P.fnp,
              s.stream);
    return 0.0;
}

void solver_compute_forces_tot(void) { total_forces(parts(), sys().stream); }

void integrator_part_1(void) {
    System& s = sys();
    if (!s.integ_ready) fatal("solver_initialize_integrator() has not been called");
    mzb::integrator_part1(parts(), s.I, s.stream);
}

void integrator_part_2(void) {
    System& s = sys();
    if (!s.integ_ready) fatal("solver_initialize_integrator() has not been called");
    mzb::integrator_part2(parts(), s.I, s.stream);
}

double get_temperature(void);

int solver_check_thermostat(void) {  // solver_md.c:210-221
    System& s = sys();
    int res = 0;
    if (s.I.enabled == 1) {
        const double temp = get_temperature();
        if (fabs(temp - s.I.T) < 100) {
            res = 1;
            s.I.enabled = 0;
            touch(s);
            if (s.I.type == 0) {
                s.I.c1 = 1.0;
                s.I.c2 = 1.0;
            }
        }
    }
    return res;
}

void solver_rescale_velocities(void) { mzb::rescale_velocities(parts(), sys().stream); }

void solver_finalize(void) {
    if (!g) return;
    touch(*g);
    if (g->stream) cudaStreamSynchronize(g->stream);
    if (g->G.ready) free_grid(g->G);
    if (g->parts_ready) free_particles(g->P);
    g->parts_ready = false;
    g->integ_ready = false;
}

// ---------------------------------------------------------------- getters (solver_md.c:247-354)
static void d2h(void* dst, const void* src, size_t bytes) {
    System& s = sys();
    if (bytes == 0) return;
    MZB_CHECK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s.stream));
    sync();
}

void get_pos(double* recv) { ParticleDev& P = parts(); d2h(recv, P.pos, sizeof(double) * 3 * P.np); }
void get_vel(double* recv) { ParticleDev& P = parts(); d2h(recv, P.vel, sizeof(double) * 3 * P.np); }
void get_fcs_elec(double* recv) { ParticleDev& P = parts(); d2h(recv, P.fe, sizeof(double) * 3 * P.np); }
void get_fcs_noel(double* recv) { ParticleDev& P = parts(); d2h(recv, P.fn, sizeof(double) * 3 * P.np); }
void get_fcs_tot(double* recv) { ParticleDev& P = parts(); d2h(recv, P.ft, sizeof(double) * 3 * P.np); }
static void get_or_zero(double* recv, const double* d, size_t count) {
    if (d) d2h(recv, d, sizeof(double) * count);
    else memset(recv, 0, sizeof(double) * count);
}
void get_fcs_db(double* recv) { ParticleDev& P = parts(); get_or_zero(recv, P.fdb, (size_t)3 * P.np); }
void get_fcs_ib(double* recv) { ParticleDev& P = parts(); get_or_zero(recv, P.fib, (size_t)3 * P.np); }
void get_fcs_np(double* recv) { ParticleDev& P = parts(); get_or_zero(recv, P.fnp, (size_t)3 * P.np); }
void get_types(int* recv) { ParticleDev& P = parts(); d2h(recv, P.types, sizeof(int32_t) * P.np); }
void get_charges(double* recv) { ParticleDev& P = parts(); d2h(recv, P.chg, sizeof(double) * P.np); }
void get_masses(double* recv) { ParticleDev& P = parts(); d2h(recv, P.mass, sizeof(double) * P.np); }
void get_radii(double* recv) { ParticleDev& P = parts(); get_or_zero(recv, P.radii, (size_t)P.np); }
void get_field(double* recv) { GridState& G = grid(); d2h(recv, G.phi(), sizeof(double) * G.m); }
void get_field_prev(double* recv) {
    GridState& G = grid();
    d2h(recv, G.type == G_FFT ? G.phi() : G.phi_prev(), sizeof(double) * G.m);
}
void get_q(double* recv) { GridState& G = grid(); d2h(recv, G.q, sizeof(double) * G.m); }

double get_kinetic_energy(void) {
    System& s = sys();
    ParticleDev& P = parts();
    kinetic_and_momentum(P, s.stream);
    d2h(s.red_h, P.red, sizeof(double) * 8);
    return s.red_h[2];
}

double get_temperature(void) {  // particles.c:798-800
    System& s = sys();
    ParticleDev& P = parts();
    kinetic_and_momentum(P, s.stream);
    d2h(s.red_h, P.red, sizeof(double) * 8);
    return s.red_h[6];
}

void get_momentum(double* recv) {
    System& s = sys();
    ParticleDev& P = parts();
    kinetic_and_momentum(P, s.stream);
    d2h(s.red_h, P.red, sizeof(double) * 8);
    recv[0] = s.red_h[3];
    recv[1] = s.red_h[4];
    recv[2] = s.red_h[5];
}


// grid_general.c:304-315: sum of 0.5*phi over the grid (what the reference computes)
double get_energy_elec(void);

}  // extern "C"

// ====================================================================================
// Extensions (no reference counterpart): kernel-level entry points on plain n^3 host
// arrays for parity tests, accessors for the linked cells / CIC corners / O-block noise,
// and a multi-step driver.
// ====================================================================================
namespace mzb {
namespace {

__global__ void k_half_sum(const double* __restrict__ phi, long m, double* __restrict__ part) {
    double v[1] = {0.0};
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (long)gridDim.x * blockDim.x)
        v[0] += 0.5 * phi[t];
    __shared__ double sh[4 * 32];
    block_sum<1>(v, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}
__global__ void k_sum_parts(const double* __restrict__ part, int nb, double* __restrict__ out) {
    double s = 0.0;
    for (int b = 0; b < nb; b++) s += part[b];
    *out = s;
}

// Stencil points of every ion in the reference's neighbour layout: CIC corners
// (particles.c:297-346) or the 64 B-spline points (particles.c:348-385).
__global__ void k_stencil_points(const int32_t* __restrict__ base, int np, int n, int cas,
                                 int64_t* __restrict__ out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const int* b = base + 3 * p;
    if (cas == CAS_CIC) {
        const int off[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}};
        for (int c = 0; c < 8; c++)
            for (int d = 0; d < 3; d++) out[(p * 8 + c) * 3 + d] = off[c][d] ? wrap_inc(b[d], n) : b[d];
    } else {
        for (int o = 0; o < 64; o++) {
            out[(p * 64 + o) * 3 + 0] = (b[0] + o / 16 - 1 + n) % n;
            out[(p * 64 + o) * 3 + 1] = (b[1] + (o / 4) % 4 - 1 + n) % n;
            out[(p * 64 + o) * 3 + 2] = (b[2] + o % 4 - 1 + n) % n;
        }
    }
}

// Temporary device work set for the kernel-level entry points.
struct Work {
    std::vector<double*> bufs;
    void* halo = nullptr;
    double* get(size_t count) {
        double* p = dalloc<double>(count);
        bufs.push_back(p);
        return p;
    }
    // The resident kernels' work area (null: n is not theirs), for the entry points that solve. It
    // goes back to the block cache: allocated and freed in each call it took 0.45 of the 1.65 ms
    // of a 30^3 call, and the other entry points paid for it too.
    void* get_halo(int n) {
        if (const size_t bytes = resident_halo_bytes(n)) halo = dalloc<unsigned char>(bytes);
        return halo;
    }
    ~Work() {
        for (double* p : bufs) cudaFree(p);
        dev_free(halo);
    }
};

EngineArgs scratch_engine(System& s, Work& w, int n) {
    const long m = (long)n * n * n, mc = m / 8 > 0 ? m / 8 : 1;
    EngineArgs a{};
    a.n = n;
    a.r = w.get(m); a.p0 = w.get(m); a.p1 = w.get(m); a.Ap = w.get(m); a.v = w.get(m); a.rf = w.get(m);
    a.tmp = w.get(m);
    a.rc = w.get(mc); a.ec = w.get(mc); a.cr = w.get(mc); a.cp0 = w.get(mc); a.cp1 = w.get(mc);
    a.cAp = w.get(mc);
    a.partials = s.partials;
    a.bar = s.bar;
    a.result = s.result;
    return a;
}

void h2d(double* d, const double* h, long m) {
    upload(d, h, sizeof(double) * m);
}
void d2h_sync(double* h, const double* d, long m) {
    MZB_CHECK(cudaMemcpy(h, d, sizeof(double) * m, cudaMemcpyDeviceToHost));
}

}  // namespace
}  // namespace mzb

extern "C" {

double get_energy_elec(void) {
    System& s = sys();
    GridState& G = grid();
    const int nb = 256;
    count_launch();
    k_half_sum<<<nb, 256, 0, s.stream>>>(G.phi(), G.m, s.scratch_d);
    count_launch();
    k_sum_parts<<<1, 1, 0, s.stream>>>(s.scratch_d, nb, s.scratch_d + nb);
    MZB_CHECK(cudaGetLastError());
    double out = 0.0;
    MZB_CHECK(cudaMemcpyAsync(s.red_h, s.scratch_d + nb, sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    sync();
    out = s.red_h[0];
    return out;
}

// out = L u (laplace.c:24-75) on plain n^3 arrays
void mzb_laplace(const double* u, double* out, int n) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    double* du = w.get(m);
    double* dout = w.get(m);
    h2d(du, u, m);
    a.prog = PROG_LAPLACE;
    a.u = du;
    a.out = dout;
    run_engine(s, a);
    d2h_sync(out, dout, m);
}

// conj_grad (plcg.c:28-90) and conj_grad_precond (plcg.c:104-166, precond 1 = JACOBI,
// 2 = MG, 3 = SSOR, 4 = BLOCKJACOBI); returns the reference's return value.
int mzb_conj_grad(const double* b, const double* x0, double* x, double tol, int n, int precond) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    if (precond == 2) require_mg_size(n);
    EngineArgs a = scratch_engine(s, w, n);
    double* db = w.get(m);
    double* dx0 = w.get(m);
    double* dx = w.get(m);
    h2d(db, b, m);
    h2d(dx0, x0, m);
    a.prog = precond == 0 ? PROG_CG : PROG_PCG;
    a.precond = precond;
    if (precond <= 1) a.halo = w.get_halo(n);
    a.tol = tol;
    a.b = db;
    a.x0 = dx0;
    a.x = dx;
    double* inv = nullptr;
    if (precond == PC_BLOCKJACOBI) {
        if (n % kBlockJacobiB) fatal("mzb_conj_grad: block Jacobi needs n to be a multiple of 10");
        a.bj_inv = inv = device_block_inverse();
    }
    const int res = run_engine(s, a);
    d2h_sync(x, dx, m);
    if (inv) cudaFree(inv);
    return res;
}

// smooth_rbgs (multigrid.c:636-729): `iters` red-black iterations on x in place
void mzb_smooth_rbgs(const double* rhs, double* x, int n, int iters) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    double* db = w.get(m);
    double* dx = w.get(m);
    h2d(db, rhs, m);
    h2d(dx, x, m);
    a.prog = PROG_SMOOTH;
    a.sm = iters;
    a.b = db;
    a.x = dx;
    run_engine(s, a);
    d2h_sync(x, dx, m);
}

// precond_blockjacobi_apply (precond_blockjacobi.c:173-206), n a multiple of 10
void mzb_blockjacobi_apply(const double* u, double* out, int n) {
    System& s = sys();
    Work w;
    if (n % kBlockJacobiB) fatal("mzb_blockjacobi_apply: n must be a multiple of 10");
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    double* du = w.get(m);
    double* dout = w.get(m);
    h2d(du, u, m);
    double* inv = device_block_inverse();
    a.prog = PROG_BLOCKJACOBI;
    a.bj_inv = inv;
    a.u = du;
    a.out = dout;
    run_engine(s, a);
    d2h_sync(out, dout, m);
    cudaFree(inv);
}

// precond_ssor_apply (precond_ssor.c:1240-1252): out = SSOR preconditioner applied to u
void mzb_ssor_apply(const double* u, double* out, int n) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    double* du = w.get(m);
    double* dout = w.get(m);
    h2d(du, u, m);
    a.prog = PROG_SSOR;
    a.u = du;
    a.out = dout;
    run_engine(s, a);
    d2h_sync(out, dout, m);
}

// restriction_27pt (multigrid.c:523-594): fine n^3 -> coarse (n/2)^3
void mzb_restrict27(const double* fine, double* coarse, int n) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    double* du = w.get(m);
    double* dout = w.get(m / 8);
    h2d(du, fine, m);
    a.prog = PROG_RESTRICT;
    a.u = du;
    a.out = dout;
    run_engine(s, a);
    d2h_sync(coarse, dout, m / 8);
}

// prolong_trilinear (multigrid.c:393-463): coarse nc^3 -> fine (2nc)^3
void mzb_prolong_trilinear(const double* coarse, double* fine, int nc) {
    System& s = sys();
    Work w;
    const long mc = (long)nc * nc * nc;
    EngineArgs a = scratch_engine(s, w, nc);
    double* du = w.get(mc);
    double* dout = w.get(mc * 8);
    h2d(du, coarse, mc);
    a.prog = PROG_PROLONG;
    a.u = du;
    a.out = dout;
    run_engine(s, a);
    d2h_sync(fine, dout, mc * 8);
}

// cg_coarse (multigrid.c:13-96); x holds the initial guess and receives the result
int mzb_cg_coarse(const double* b, double* x, int n, int maxit, double rtol) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    double* db = w.get(m);
    double* dx = w.get(m);
    h2d(db, b, m);
    h2d(dx, x, m);
    a.prog = PROG_CG_COARSE;
    a.maxit = maxit;
    a.rtol = rtol;
    a.b = db;
    a.x0 = dx;
    a.x = dx;
    const int res = run_engine(s, a);
    d2h_sync(x, dx, m);
    return res;
}

// one V-cycle (multigrid.c:99-168) with `sm` RBGS iterations per half; x in place
void mzb_mg_apply(const double* rhs, double* x, int n, int sm) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    require_mg_size(n);
    EngineArgs a = scratch_engine(s, w, n);
    double* db = w.get(m);
    double* dx = w.get(m);
    h2d(db, rhs, m);
    h2d(dx, x, m);
    a.prog = PROG_MG_APPLY;
    a.sm = sm;
    a.b = db;
    a.x = dx;
    run_engine(s, a);
    d2h_sync(x, dx, m);
}

// ---- Poisson-Boltzmann kernel-level entry points: ex/ey/ez/k2 are host n^3 arrays of the
// +x/+y/+z face coefficients and screening term of each point.
}  // extern "C"
namespace mzb {
namespace {
PbGrid scratch_pb(System& s, Work& w, int n, const double* ex, const double* ey, const double* ez,
                  const double* k2, bool coarse) {
    const long m = (long)n * n * n;
    PbGrid g;
    g.n = n;
    g.ex = w.get(m); g.ey = w.get(m); g.ez = w.get(m); g.k2 = w.get(m); g.dg = w.get(m);
    h2d(g.ex, ex, m); h2d(g.ey, ey, m); h2d(g.ez, ez, m); h2d(g.k2, k2, m);
    if (coarse) {
        const long mc = m / 8;
        g.cex = w.get(mc); g.cey = w.get(mc); g.cez = w.get(mc); g.ck2 = w.get(mc); g.cdg = w.get(mc);
    }
    pb_derive(g, s.stream);
    return g;
}
}  // namespace
}  // namespace mzb
extern "C" {

// out = A_pb u (laplace.c:77-145)
void mzb_laplace_pb(const double* u, double* out, const double* ex, const double* ey, const double* ez,
                    const double* k2, int n) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    set_pb_operator(a, scratch_pb(s, w, n, ex, ey, ez, k2, false));
    double* du = w.get(m);
    double* dout = w.get(m);
    h2d(du, u, m);
    a.prog = PROG_LAPLACE;
    a.u = du;
    a.out = dout;
    run_engine(s, a);
    d2h_sync(out, dout, m);
}

// conj_grad_pb (plcg.c:169-238); returns the reference's return value
int mzb_conj_grad_pb(const double* b, const double* x0, double* x, double tol, int n, const double* ex,
                     const double* ey, const double* ez, const double* k2) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    set_pb_operator(a, scratch_pb(s, w, n, ex, ey, ez, k2, false));
    double* db = w.get(m);
    double* dx0 = w.get(m);
    double* dx = w.get(m);
    h2d(db, b, m);
    h2d(dx0, x0, m);
    a.prog = PROG_CG;
    a.halo = w.get_halo(n);
    a.tol = tol;
    a.b = db;
    a.x0 = dx0;
    a.x = dx;
    const int res = run_engine(s, a);
    d2h_sync(x, dx, m);
    return res;
}

// smooth_pb_rbgs (multigrid_pb.c:544-640): `iters` red-black iterations on x in place
void mzb_smooth_pb(const double* rhs, double* x, int n, int iters, const double* ex, const double* ey,
                   const double* ez, const double* k2) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    EngineArgs a = scratch_engine(s, w, n);
    set_pb_operator(a, scratch_pb(s, w, n, ex, ey, ez, k2, false));
    double* db = w.get(m);
    double* dx = w.get(m);
    h2d(db, rhs, m);
    h2d(dx, x, m);
    a.prog = PROG_SMOOTH;
    a.sm = iters;
    a.b = db;
    a.x = dx;
    run_engine(s, a);
    d2h_sync(x, dx, m);
}

// one PB V-cycle (multigrid_pb.c:270-328) with `sm` smoother iterations per half; x in place
void mzb_mg_pb_apply(const double* rhs, double* x, int n, int sm, const double* ex, const double* ey,
                     const double* ez, const double* k2) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    require_mg_size(n);
    EngineArgs a = scratch_engine(s, w, n);
    set_pb_operator(a, scratch_pb(s, w, n, ex, ey, ez, k2, true));
    double* db = w.get(m);
    double* dx = w.get(m);
    h2d(db, rhs, m);
    h2d(dx, x, m);
    a.prog = PROG_MG_APPLY;
    a.sm = sm;
    a.b = db;
    a.x = dx;
    run_engine(s, a);
    d2h_sync(x, dx, m);
}

// coarse coefficients of the PB V-cycle (restriction_eps, restriction_k2screen,
// multigrid_pb.c:330-527): (n/2)^3 outputs
void mzb_restrict_pb(const double* ex, const double* ey, const double* ez, const double* k2, double* cex,
                     double* cey, double* cez, double* ck2, int n) {
    System& s = sys();
    Work w;
    const PbGrid g = scratch_pb(s, w, n, ex, ey, ez, k2, true);
    MZB_CHECK(cudaStreamSynchronize(s.stream));
    const long mc = (long)(n / 2) * (n / 2) * (n / 2);
    d2h_sync(cex, g.cex, mc);
    d2h_sync(cey, g.cey, mc);
    d2h_sync(cez, g.cez, mc);
    d2h_sync(ck2, g.ck2, mc);
}

// The PB coefficients of the current grid (after solver_update_eps_k2).
void mzb_get_pb_grids(double* ex, double* ey, double* ez, double* k2) {
    System& s = sys();
    GridState& G = grid();
    if (!G.pb) fatal("mzb_get_pb_grids: the grid has no Poisson-Boltzmann coefficients");
    MZB_CHECK(cudaStreamSynchronize(s.stream));
    d2h_sync(ex, G.pbg.ex, G.m);
    d2h_sync(ey, G.pbg.ey, G.m);
    d2h_sync(ez, G.pbg.ez, G.m);
    d2h_sync(k2, G.pbg.k2, G.m);
}

// rfft_solve with the reference's ig2 (grid_fft.c:65-125, fftw_wrap.c:166-189)
void mzb_fft_poisson(const double* q, double* phi, int n, double L, double h) {
    System& s = sys();
    Work w;
    const long m = (long)n * n * n;
    double* dq = w.get(m);
    double* dphi = w.get(m);
    h2d(dq, q, m);
    FftPoisson f;
    f.init(n, L, h);
    f.solve(dq, dphi, s.stream);
    sync();
    f.release();
    d2h_sync(phi, dphi, m);
}

// Stencil (neighbour) indices of the current system in the reference's layout: (n_p, 8, 3)
// int64 for CIC (particles.c:297-346), (n_p, 64, 3) for the B-splines
// (particles.c:348-385); valid after solver_update_charges.
void mzb_get_cic_neighbors(int64_t* out) {
    System& s = sys();
    ParticleDev& P = parts();
    if (P.np == 0) return;
    const int nnb = P.cas == CAS_CIC ? 8 : 64;
    int64_t* d = nullptr;
    MZB_CHECK(cudaMalloc(&d, sizeof(int64_t) * 3 * nnb * P.np));
    count_launch();
    k_stencil_points<<<(P.np + 127) / 128, 128, 0, s.stream>>>(P.base, P.np, grid().n, P.cas, d);
    MZB_CHECK(cudaMemcpyAsync(out, d, sizeof(int64_t) * 3 * nnb * P.np, cudaMemcpyDeviceToHost, s.stream));
    sync();
    cudaFree(d);
}

// Linked cells per side used by the pair-force kernel (default ~16 ions per cell).
void mzb_set_cell_grid(int nc) {
    ParticleDev& P = parts();
    sync();
    set_cells(P, nc);
    touch(sys());
}

// Build the linked cells for the current positions and copy them out: start has
// nc^3 + 1 entries, ions n_p. Returns nc.
int mzb_get_cells(int32_t* start, int32_t* ions) {
    System& s = sys();
    ParticleDev& P = parts();
    build_cells(P, s.stream);
    MZB_CHECK(cudaMemcpyAsync(start, P.cell_start, sizeof(int32_t) * (P.ncell + 1), cudaMemcpyDeviceToHost,
                              s.stream));
    if (P.np > 0)
        MZB_CHECK(cudaMemcpyAsync(ions, P.cell_ions, sizeof(int32_t) * P.np, cudaMemcpyDeviceToHost, s.stream));
    sync();
    return P.nc;
}

// O-block noise: the N(0,1) draws the O-block applies on its `call`-th application
// (integrator_ovrvo.c:45-78 draws them from glibc rand()), 3*n_p values.
void mzb_philox_normals(uint64_t call, double* out) {
    System& s = sys();
    ParticleDev& P = parts();
    if (P.np == 0) return;
    double* d = nullptr;
    MZB_CHECK(cudaMalloc(&d, sizeof(double) * 3 * P.np));
    philox_normals(s.I.seed, call, P.np, d, s.stream);
    MZB_CHECK(cudaMemcpyAsync(out, d, sizeof(double) * 3 * P.np, cudaMemcpyDeviceToHost, s.stream));
    sync();
    cudaFree(d);
}

void mzb_set_seed(uint64_t seed) {
    sys().I.seed = seed;
    touch(sys());
}

// Field-solve form of the current grid: 0 = the reference's FP64 algorithms, 1 = FP32
// multigrid with FP64 iterative refinement to the same (or an overriding) tolerance, 2 =
// the same multigrid with every value in FP64 (the FP64 multigrid form). Grids that cannot
// be coarsened three times, and FFT, stay on the reference's algorithms.
void mzb_set_precision(int mode, double tol_override) {
    GridState& G = grid();
    touch(sys());
    G.precision = (mode == 1 || mode == 2) ? mode : 0;
    G.mixed_tol = tol_override;
}
int mzb_get_precision(void) {
    GridState& G = grid();
    return (G.precision >= 1 && mixed_supported(G)) ? G.precision : 0;
}

// Coarse-level plan of the current grid's multigrid forms (precision 1 and 2): 0 = the
// levels go down to the first one of at most 16 points per side, solved by its Green's
// function; 1 or 2 = the first level from level 1 or 2 on with 32, 64 or 128 points per side
// is the coarse level, solved by FFT; -1 = the default (1). mzb_batch_autotune sets it per
// size class. Returns -1 for an unknown plan.
int mzb_set_mixed_plan(int plan) {
    if (plan < -1 || plan > 2) return -1;
    GridState& G = grid();
    touch(sys());
    G.plan = plan;
    return 0;
}
// The level the current grid's multigrid forms solve by FFT (1, 2), or 0 when the coarsest
// level is solved by its Green's function (or the grid has no multigrid form).
int mzb_get_mixed_plan(void) {
    GridState& G = grid();
    if (!(G.precision >= 1 && mixed_supported(G))) return 0;
    ensure_mixed_levels(G);
    return G.coarse_fft ? G.nlev - 1 : 0;
}

// Red-black Gauss-Seidel sweeps before (nu1) and after (nu2) the coarse correction of the
// current grid's multigrid forms; 1 .. 16 each.
int mzb_set_mixed_sweeps(int nu1, int nu2) {
    if (nu1 < 1 || nu1 > 16 || nu2 < 1 || nu2 > 16) return -1;
    GridState& G = grid();
    touch(sys());
    G.nu1 = nu1;
    G.nu2 = nu2;
    return 0;
}
void mzb_get_mixed_sweeps(int* nu1, int* nu2) {
    GridState& G = grid();
    if (nu1) *nu1 = G.nu1;
    if (nu2) *nu2 = G.nu2;
}

// The CUDA stream all work of the current system is queued on (for callers that time
// it with their own events or order their own kernels against it).
void* mzb_get_stream(void) { return (void*)sys().stream; }

// Device time (CUDA events on the library stream) and return value of the last
// field-solver launch (one solver_update_field / solver_init_field).
double mzb_last_solve_ms(void) { return (double)sys().last_solve_ms; }
int mzb_last_solve_result(void) { return sys().last_solve_iters; }

// Kernels launched by this library since it was loaded.
uint64_t mzb_kernel_launches(void) { return g_kernel_launches; }
int mzb_sm_count(void) { return mixed_grid_blocks(); }
// Green's function of the unscaled periodic 7-point Laplacian on an n^3 grid (its
// pseudo-inverse; the mixed solver's coarsest level is solved with it): g[0..n^3).
int mzb_coarse_green(int n, float* g) {
    if (n < 2 || n > kMixedTeamDirectN || !g) return -1;
    mixed_coarse_green(n, g);
    return 0;
}
uint64_t mzb_get_ocalls(void) { return sys().I.ocalls; }

// n_steps iterations of SolverMD.md_loop_iter (maze_poisson/solver.py:483-492) with both
// electrostatic and non-electrostatic forces (and the PB coefficient update and forces on
// a Poisson-Boltzmann grid); returns the last solver_update_field value. Poisson grids
// (every method and form) run the steps without a host round trip:
// the charge check and the solve status stay on the device and are read after the last
// step (md_steps_deferred); a charge error still prints the reference's message and exits.
int solver_md_step(int n_steps) {
    if (n_steps <= 0) return 0;
    {
        System& s = sys();
        GridState& G = grid();
        if (!G.pb && !(G.type == G_MAZE_MG && G.precond != P_NONE) && s.parts_ready && s.integ_ready)
            return md_steps_deferred(s, n_steps);
    }
    int res = 0;
    for (int i = 0; i < n_steps; i++) {
        const bool pb = grid().pb;
        integrator_part_1();
        solver_update_charges();
        if (pb) solver_update_eps_k2();
        res = solver_update_field();
        solver_compute_forces_elec();
        solver_compute_forces_noel();
        if (pb) solver_compute_forces_pb();
        solver_compute_forces_tot();
        integrator_part_2();
    }
    sync();
    return res;
}

}  // extern "C"

// ====================================================================================
// Several resident systems and the batched step (this build's extension; the reference
// holds one system per process, solver_md.c:12-14).
//
// A system handle selects which system the reference-ABI calls act on. mzb_batch_step
// advances a set of systems together: per MD step one CUDA graph forks a branch per
// system for integrator part 1 + charge spreading (+ a device-side charge check), joins
// into ONE cooperative launch that runs every system's mixed-precision field solve on its
// own range of CTAs (mixed_batch_kernel), and forks again for field + pair + total forces
// and integrator part 2. The graph bakes in each system's buffer pointers, which rotate
// with period 3 after every solve, so up to three graphs per membership are cached.
// mzb_batch_classes runs several such batches (size classes) side by side, each on its
// own stream with its own share of the CTAs and its own number of steps per call.
// ====================================================================================
namespace mzb {
namespace {

__global__ void k_charge_check(const double* red, double* qtot, int* err) {
    const double q = red[0];
    if (fabs(*qtot - q) > 1e-6) err[0] = 1;  // solver_md.c:98-102
    *qtot = q;
}
__global__ void k_solve_check(const int* result, int* err) {
    if (result[0] < 0 || result[1] != 0) err[2] = 1;
}

struct BatchGraph {
    std::vector<uint64_t> key;
    std::vector<int> handles;
    cudaGraphExec_t exec = nullptr;
    MixedArgs* list_d = nullptr;
    int* start_d = nullptr;
    StageTable stages;  // replica table of the particle stages (nsys 0: per-system branches)
    unsigned long long launches = 0;
    unsigned long long used = 0;  // call counter of the last use (least recently used goes first)
};

struct Batch {
    int device = -1;
    cudaEvent_t fork1 = nullptr, fork2 = nullptr, t0 = nullptr, t1 = nullptr;
    std::vector<cudaStream_t> streams;  // one per size class; streams[0] also serves mzb_batch_step
    std::vector<cudaEvent_t> join1, join2;
    std::vector<BatchGraph> graphs;
    size_t capacity = 6;
    unsigned long long calls = 0;
    double alpha = 1.0;  // team size ~ (grid points)^alpha (autotuned)
};
Batch g_batchst;
// MZB_BATCH_BRANCHES=1 (a comparison aid): the particle stages as one graph branch per
// system instead of replica tables
const bool g_batch_branches = getenv("MZB_BATCH_BRANCHES") != nullptr && strcmp(getenv("MZB_BATCH_BRANCHES"), "0") != 0;

void release_graph(BatchGraph& bg) {
    if (bg.exec) cudaGraphExecDestroy(bg.exec);
    dev_free(bg.list_d);
    dev_free(bg.start_d);
    if (bg.stages.nsys) stage_table_free(bg.stages);
    bg = BatchGraph{};
}

void batch_clear_graphs() {
    for (auto& bg : g_batchst.graphs) release_graph(bg);
    g_batchst.graphs.clear();
}

// Release the graphs that step system `handle` (the others stay valid).
void batch_drop_graphs(int handle) {
    auto& gs = g_batchst.graphs;
    for (size_t i = 0; i < gs.size();) {
        if (std::find(gs[i].handles.begin(), gs[i].handles.end(), handle) != gs[i].handles.end()) {
            release_graph(gs[i]);
            gs.erase(gs.begin() + i);
        } else {
            i++;
        }
    }
}

void batch_events(int nsys, int nclass = 1) {
    Batch& B = g_batchst;
    int dev;
    MZB_CHECK(cudaGetDevice(&dev));
    if (B.device != dev) {
        MZB_CHECK(cudaEventCreateWithFlags(&B.fork1, cudaEventDisableTiming));
        MZB_CHECK(cudaEventCreateWithFlags(&B.fork2, cudaEventDisableTiming));
        MZB_CHECK(cudaEventCreate(&B.t0));
        MZB_CHECK(cudaEventCreate(&B.t1));
        B.device = dev;
    }
    while ((int)B.streams.size() < nclass) {
        cudaStream_t st;
        MZB_CHECK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        B.streams.push_back(st);
    }
    while ((int)B.join1.size() < nsys) {
        cudaEvent_t e1, e2;
        MZB_CHECK(cudaEventCreateWithFlags(&e1, cudaEventDisableTiming));
        MZB_CHECK(cudaEventCreateWithFlags(&e2, cudaEventDisableTiming));
        B.join1.push_back(e1);
        B.join2.push_back(e2);
    }
}

System& checked_system(int h) {
    if (h < 0 || h >= (int)g_systems.size() || !g_systems[h]) fatal("batched step: invalid system handle");
    System& s = *g_systems[h];
    if (!s.G.ready || !s.parts_ready || !s.integ_ready) fatal("batched step: system is not fully initialised");
    if (s.G.type == G_FFT || s.G.precision != 1 || !mixed_supported(s.G))
        fatal("batched step: every system must use the mixed-precision (FP32+refine) field solve");
    return s;
}

// Device-side state a batched step needs (charge total, error flags, Philox counter).
void batch_prepare(System& s) {
    if (!s.qtot_d) {
        s.qtot_d = dalloc<double>(1);
        s.err_d = dalloc<int>(4);
        zero_fill(s.err_d, 4 * sizeof(int));
    }
    if (!s.I.ocalls_d) {
        s.I.ocalls_d = dalloc<uint64_t>(1);
        touch(s);
    }
    upload(s.qtot_d, &s.q_tot, sizeof(double));
    upload(s.I.ocalls_d, &s.I.ocalls, sizeof(uint64_t));
}

// Team partition of nblocks CTAs: at least one per system, the rest in proportion to
// (grid points)^alpha times the system's cost factor (1 without the tuner's factors) by
// largest remainder.
std::vector<int> team_starts(const std::vector<System*>& ss, int nblocks, double alpha) {
    const int n = (int)ss.size();
    std::vector<double> w(n);
    double tot = 0.0;
    for (int r = 0; r < n; r++) {
        w[r] = pow((double)ss[r]->G.m, alpha) * ss[r]->G.batch_cost;
        tot += w[r];
    }
    const int rem = nblocks - n;
    std::vector<int> cnt(n, 1);
    std::vector<std::pair<double, int>> frac(n);
    int used = 0;
    for (int r = 0; r < n; r++) {
        const double share = rem * w[r] / tot;
        const int f = (int)floor(share);
        cnt[r] += f;
        used += f;
        frac[r] = {share - f, r};
    }
    std::sort(frac.begin(), frac.end(), [](const std::pair<double, int>& a, const std::pair<double, int>& b) {
        return a.first > b.first || (a.first == b.first && a.second < b.second);
    });
    for (int k = 0; used < rem; k++, used++) cnt[frac[k % n].second]++;
    std::vector<int> start(n + 1, 0);
    for (int r = 0; r < n; r++) start[r + 1] = start[r] + cnt[r];
    return start;
}

// The particle stages' arguments of system s in a batched step (replica tables).
StageArgs stage_args(System& s) {
    StageArgs a;
    a.P = s.P;
    a.I = s.I;
    a.q = s.G.q;
    a.qmask = s.G.qmask;
    a.n = s.G.n;
    a.h = s.G.h;
    a.mask_words = s.G.qmask != nullptr ? (int)(((size_t)s.G.n * s.G.n * (s.G.n >> 6) + 31) / 32) : 0;
    a.q_sparse = s.P.cas == CAS_CIC && s.P.q_sparse == s.G.q ? 1 : 0;
    a.phi = s.G.buf[s.G.ispare];  // the field the solve writes
    a.qtot = s.qtot_d;
    a.err = s.err_d;
    a.result = s.result;
    a.bar = s.bar;
    return a;
}

void stage_particles_before_solve(System& s) {
    ParticleDev& P = s.P;
    integrator_part1(P, s.I, s.stream);
    spread_charges(P, s.G.q, s.G.qmask, s.G.n, s.G.h, s.stream);
    count_launch();
    k_charge_check<<<1, 1, 0, s.stream>>>(P.red, s.qtot_d, s.err_d);
}

void stage_particles_after_solve(System& s) {
    ParticleDev& P = s.P;
    count_launch();
    k_solve_check<<<1, 1, 0, s.stream>>>(s.result, s.err_d);
    field_forces(P, s.G.buf[s.G.ispare], s.G.n, s.G.h, s.stream);  // the field the solve wrote
    build_cells(P, s.stream);
    tf_forces(P, s.stream);
    total_forces(P, s.stream);
    integrator_part2(P, s.I, s.stream);
}

__global__ void k_md_charge_check(const double* red, double* qtot, int* err, double* bad) {
    const double q = red[0];
    if (fabs(*qtot - q) > 1e-6 && !err[0]) {  // solver_md.c:98-102, first failing step kept
        err[0] = 1;
        bad[0] = *qtot;
        bad[1] = q;
    }
    *qtot = q;
}

// solver_md_step on a Poisson grid without host round trips: per step integrator part 1,
// spreading with the charge check on the device, the field solve launched without reading
// its result (the buffers rotate as solver_update_field rotates them), field, pair and
// total forces, integrator part 2. One synchronisation at the end reads the error words,
// the charge total and the last solve's result and time.
int md_steps_deferred(System& s, int n_steps) {
    GridState& G = s.G;
    ParticleDev& P = s.P;
    batch_prepare(s);  // device charge total, error words, Philox counter
    double* bad = s.scratch_d + 4094;  // the last two words of the 4096-double scratch
    for (int i = 0; i < n_steps; i++) {
        integrator_part1(P, s.I, s.stream);
        spread_charges(P, G.q, G.qmask, G.n, G.h, s.stream);
        count_launch();
        k_md_charge_check<<<1, 1, 0, s.stream>>>(P.red, s.qtot_d, s.err_d, bad);
        MZB_CHECK(cudaEventRecord(s.ev0, s.stream));
        if (G.type == G_FFT) {  // in place, no previous field, no status word
            G.fft.solve(G.q, G.phi(), s.stream);
            MZB_CHECK(cudaEventRecord(s.ev1, s.stream));
        } else {
            if (G.precision >= 1 && mixed_supported(G)) {
                double cst = 0.0;
                const int prog = mixed_update_prog(G, cst);
                mixed_launch(mixed_args(s, prog, cst), s.stream);
            } else {
                launch_solver(update_engine_args(s), s.stream);
            }
            MZB_CHECK(cudaEventRecord(s.ev1, s.stream));
            const int old = G.iphi;
            G.iphi = G.ispare;
            G.ispare = G.iprev;
            G.iprev = old;
            count_launch();
            k_solve_check<<<1, 1, 0, s.stream>>>(s.result, s.err_d);
        }
        field_forces(P, G.phi(), G.n, G.h, s.stream);
        build_cells(P, s.stream);
        tf_forces(P, s.stream);
        total_forces(P, s.stream);
        integrator_part2(P, s.I, s.stream);
    }
    int err[4];
    double q = 0.0, qbad[2] = {0.0, 0.0};
    if (G.type == G_FFT) {
        s.result_h[0] = 0;
        s.result_h[1] = 0;
    } else {
        MZB_CHECK(cudaMemcpyAsync(s.result_h, s.result, 2 * sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    }
    MZB_CHECK(cudaStreamSynchronize(s.stream));
    MZB_CHECK(cudaMemcpy(err, s.err_d, sizeof(err), cudaMemcpyDeviceToHost));
    MZB_CHECK(cudaMemcpy(&q, s.qtot_d, sizeof(double), cudaMemcpyDeviceToHost));
    MZB_CHECK(cudaMemcpy(qbad, bad, sizeof(qbad), cudaMemcpyDeviceToHost));
    MZB_CHECK(cudaEventElapsedTime(&s.last_solve_ms, s.ev0, s.ev1));
    s.last_solve_iters = s.result_h[0];
    if (err[0]) {
        printf("Charge conservation error: q_tot = %.6f, q_tot_loc = %.6f\n", qbad[0], qbad[1]);
        exit(1);
    }
    s.q_tot = q;
    int res = s.result_h[0];
    if (s.result_h[1] != 0) {
        fprintf(stderr, "maze_poisson_b200: field solver aborted (grid barrier timeout)\n");
        res = -1;
    } else if (err[2]) {
        res = -1;  // an earlier step's solve did not converge
    }
    if (res == -1 && G.type == G_MAZE_MG)
        fprintf(stderr, "Warning: Multigrid did not converge after 1000 iterations.\n");
    if (err[2]) zero_fill(s.err_d, 4 * sizeof(int));
    return res;
}

// Build (or find) the graph of one batched MD step for the systems' current state, its
// field solves on `nblocks` CTAs, captured on `stream` (any stream may launch it). `first`
// is the index of the systems' first join events (each system of a call has its own).
BatchGraph& batch_graph(const std::vector<int>& handles, const std::vector<System*>& ss, int nblocks,
                        cudaStream_t stream, int first) {
    Batch& B = g_batchst;
    std::vector<uint64_t> key;
    key.push_back((uint64_t)(B.alpha * 1e6));
    key.push_back((uint64_t)nblocks);
    for (size_t r = 0; r < ss.size(); r++) {
        key.push_back((uint64_t)handles[r]);
        key.push_back(ss[r]->epoch);
        key.push_back((uint64_t)ss[r]->G.iphi);
    }
    for (auto& bg : B.graphs)
        if (bg.key == key) {
            bg.used = B.calls;
            return bg;
        }
    while (B.graphs.size() >= B.capacity) {  // least recently used first
        size_t v = 0;
        for (size_t i = 1; i < B.graphs.size(); i++)
            if (B.graphs[i].used < B.graphs[v].used) v = i;
        release_graph(B.graphs[v]);
        B.graphs.erase(B.graphs.begin() + v);
    }
    const int nsys = (int)ss.size();
    std::vector<MixedArgs> list(nsys);
    size_t smem = 0;
    for (int r = 0; r < nsys; r++) {
        double cst = 0.0;
        const int prog = mixed_update_prog(ss[r]->G, cst);
        list[r] = mixed_args(*ss[r], prog, cst);
        smem = std::max(smem, mixed_smem_bytes(list[r]));
    }
    const std::vector<int> start = team_starts(ss, nblocks, B.alpha);
    BatchGraph bg;
    bg.key = key;
    bg.handles = handles;
    bg.used = B.calls;
    bg.list_d = static_cast<MixedArgs*>(dev_alloc(sizeof(MixedArgs) * nsys));
    bg.start_d = static_cast<int*>(dev_alloc(sizeof(int) * (nsys + 1)));
    upload(bg.list_d, list.data(), sizeof(MixedArgs) * nsys);
    upload(bg.start_d, start.data(), sizeof(int) * (nsys + 1));

    // CIC systems take the particle stages as replica tables: one launch per stage for
    // all of them; otherwise each system's stages run as a branch of the graph
    std::vector<StageArgs> sargs;
    bool tables = !g_batch_branches;
    for (int r = 0; r < nsys && tables; r++) {
        sargs.push_back(stage_args(*ss[r]));
        tables = stage_table_ok(sargs.back());
    }
    if (tables) bg.stages = stage_table_build(sargs);

    const unsigned long long l0 = g_kernel_launches;
    cudaGraph_t graph = nullptr;
    MZB_CHECK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    if (tables) {
        stages_before_solve(bg.stages, stream);  // also zeroes the solve's barriers
        mixed_batch_launch(bg.list_d, bg.start_d, nsys, nblocks, smem, stream);
        stages_after_solve(bg.stages, stream);
        for (System* sp : ss) sp->P.q_sparse = sp->G.q;  // as spread_charges leaves it
    } else {
        MZB_CHECK(cudaEventRecord(B.fork1, stream));
        for (int r = 0; r < nsys; r++) {
            MZB_CHECK(cudaStreamWaitEvent(ss[r]->stream, B.fork1, 0));
            stage_particles_before_solve(*ss[r]);
            MZB_CHECK(cudaEventRecord(B.join1[first + r], ss[r]->stream));
            MZB_CHECK(cudaStreamWaitEvent(stream, B.join1[first + r], 0));
        }
        for (int r = 0; r < nsys; r++) MZB_CHECK(cudaMemsetAsync(ss[r]->bar, 0, sizeof(GridBarrier), stream));
        mixed_batch_launch(bg.list_d, bg.start_d, nsys, nblocks, smem, stream);
        MZB_CHECK(cudaEventRecord(B.fork2, stream));
        for (int r = 0; r < nsys; r++) {
            MZB_CHECK(cudaStreamWaitEvent(ss[r]->stream, B.fork2, 0));
            stage_particles_after_solve(*ss[r]);
            MZB_CHECK(cudaEventRecord(B.join2[first + r], ss[r]->stream));
            MZB_CHECK(cudaStreamWaitEvent(stream, B.join2[first + r], 0));
        }
    }
    MZB_CHECK(cudaStreamEndCapture(stream, &graph));
    bg.launches = g_kernel_launches - l0;
    g_kernel_launches = l0;  // counted when the graph runs
    MZB_CHECK(cudaGraphInstantiate(&bg.exec, graph, 0));
    MZB_CHECK(cudaGraphDestroy(graph));
    B.graphs.push_back(bg);
    return B.graphs.back();
}

std::vector<System*> batch_systems(const int* handles, int nsys) {
    if (nsys < 1) fatal("batched step: no systems");
    std::vector<System*> ss;
    for (int r = 0; r < nsys; r++) {
        System& s = checked_system(handles[r]);
        for (System* o : ss)
            if (o == &s) fatal("batched step: a system is listed twice");
        ss.push_back(&s);
    }
    if (nsys > mixed_grid_blocks()) fatal("batched step: more systems than SMs");
    return ss;
}

// Wait for the systems' own streams, set up their device-side state.
void batch_begin(std::vector<System*>& ss, int nclass = 1) {
    batch_events((int)ss.size(), nclass);
    g_batchst.calls++;
    for (System* s : ss) {
        MZB_CHECK(cudaStreamSynchronize(s->stream));
        batch_prepare(*s);
    }
}

// Wait for the batch, copy the device-side state back and report errors the way the
// per-call path does (solver_md.c:98-102 exits on a charge error).
int batch_end(std::vector<System*>& ss, const int* handles, int nclass = 1) {
    for (int c = 0; c < nclass; c++) MZB_CHECK(cudaStreamSynchronize(g_batchst.streams[c]));
    int status = 0;
    for (size_t r = 0; r < ss.size(); r++) {
        System& s = *ss[r];
        int err[4];
        double q = 0.0;
        MZB_CHECK(cudaMemcpy(err, s.err_d, sizeof(err), cudaMemcpyDeviceToHost));
        MZB_CHECK(cudaMemcpy(&q, s.qtot_d, sizeof(double), cudaMemcpyDeviceToHost));
        MZB_CHECK(cudaMemcpy(&s.I.ocalls, s.I.ocalls_d, sizeof(uint64_t), cudaMemcpyDeviceToHost));
        if (err[0]) {
            printf("Charge conservation error in system %d: q_tot = %.6f\n", handles[r], s.q_tot);
            exit(1);
        }
        if (err[2]) status = -1;
        s.q_tot = q;
        zero_fill(s.err_d, 4 * sizeof(int));
    }
    return status;
}

void rotate_fields(const std::vector<System*>& ss) {  // phi_prev <- old phi, phi <- the solve's output
    for (System* s : ss) {
        GridState& G = s->G;
        const int old = G.iphi;
        G.iphi = G.ispare;
        G.ispare = G.iprev;
        G.iprev = old;
    }
}

// Class c takes steps[c] graph launches on its own stream, interleaved across the classes
// so that every stream has work queued early. All graphs of the call (at most three
// buffer rotations per class) are built first: building one allocates device memory and
// copies on the legacy stream, which would otherwise stop the classes from overlapping.
void batch_run(const std::vector<std::vector<int>>& hv, const std::vector<std::vector<System*>>& cs,
               const std::vector<int>& ctas, const std::vector<int>& steps) {
    Batch& B = g_batchst;
    const int nclass = (int)cs.size();
    int most = 0, first = 0;
    std::vector<int> firsts(nclass);
    for (int c = 0; c < nclass; c++) {
        most = std::max(most, steps[c]);
        firsts[c] = first;
        first += (int)cs[c].size();
    }
    B.capacity = std::max<size_t>(B.capacity, 3 * (size_t)nclass + 3);
    for (int c = 0; c < nclass; c++) {
        const int k = std::min(steps[c], 3);
        for (int t = 0; t < k; t++) {
            batch_graph(hv[c], cs[c], ctas[c], B.streams[c], firsts[c]);
            rotate_fields(cs[c]);
        }
        for (int t = k; t < 3 && k > 0; t++) rotate_fields(cs[c]);  // back to the starting rotation
    }
    for (int k = 0; k < most; k++) {
        for (int c = 0; c < nclass; c++) {
            if (k >= steps[c]) continue;
            BatchGraph& bg = batch_graph(hv[c], cs[c], ctas[c], B.streams[c], firsts[c]);
            MZB_CHECK(cudaGraphLaunch(bg.exec, B.streams[c]));
            g_kernel_launches += bg.launches;
            rotate_fields(cs[c]);
        }
    }
}

void release_snapshots(int handle);  // output snapshots of a system (defined below)

}  // namespace
}  // namespace mzb

extern "C" {

// Create an empty system and select it; returns its handle. Initialise it with the
// reference calls (solver_initialize, solver_initialize_grid, ...).
int mzb_system_create(void) {
    System* s = new System();
    g_systems.push_back(s);
    g_current = (int)g_systems.size() - 1;
    g = s;
    return g_current;
}

// Make `handle` the system the reference-ABI calls act on; -1 if it does not exist.
int mzb_system_select(int handle) {
    if (handle < 0 || handle >= (int)g_systems.size() || !g_systems[handle]) return -1;
    g_current = handle;
    g = g_systems[handle];
    return 0;
}

int mzb_system_current(void) { return g_current; }

// Free a system and everything it holds on the device; -1 if it does not exist.
int mzb_system_destroy(int handle) {
    if (handle < 0 || handle >= (int)g_systems.size() || !g_systems[handle]) return -1;
    System* prev = g;
    const int prev_h = g_current;
    g = g_systems[handle];
    solver_finalize();
    System& s = *g;
    batch_drop_graphs(handle);
    if (s.stream) cudaStreamDestroy(s.stream);
    if (s.ev0) cudaEventDestroy(s.ev0);
    if (s.ev1) cudaEventDestroy(s.ev1);
    dfree(s.partials);
    dfree(s.bar);
    dfree(s.result);
    dfree(s.scratch_d);
    dfree(s.qtot_d);
    dfree(s.err_d);
    dfree(s.I.ocalls_d);
    if (s.result_h) cudaFreeHost(s.result_h);
    if (s.red_h) cudaFreeHost(s.red_h);
    release_snapshots(handle);
    delete g_systems[handle];
    g_systems[handle] = nullptr;
    if (prev_h == handle) {
        g = nullptr;
        g_current = -1;
    } else {
        g = prev;
        g_current = prev_h;
    }
    return 0;
}

// Advance the listed systems (FP32+refine field solve, set up and bootstrapped through
// the reference calls) by n_steps MD steps together, one CUDA graph per step (see the
// section comment). Returns 0, or -1 if any field solve did not converge.
int mzb_batch_step(const int* handles, int nsys, int n_steps) {
    std::vector<System*> ss = batch_systems(handles, nsys);
    batch_begin(ss);
    std::vector<int> hv(handles, handles + nsys);
    batch_run({hv}, {ss}, {mixed_grid_blocks()}, {n_steps});
    return batch_end(ss, handles);
}

// Size classes side by side: system r belongs to class cls[r] (0 <= cls[r] < nclass);
// class c advances class_steps[c] MD steps (at least 0) on its own stream, its systems'
// field solves sharing class_ctas[c] CTAs (at least one per system), while the other
// classes run theirs: the classes' kernels overlap on the device, each class at its own
// pace. The CTA counts must add up to at most the SM count, so that every class's
// cooperative solve can be resident together with the others'. Each class runs the steps
// of mzb_batch_step (the same graphs, the same results); returns when all classes are
// done: 0, or -1 if any field solve did not converge.
int mzb_batch_classes(const int* handles, const int* cls, int nsys, const int* class_ctas, const int* class_steps,
                      int nclass) {
    if (nclass < 1) fatal("batched classes: no classes");
    std::vector<System*> ss = batch_systems(handles, nsys);
    std::vector<std::vector<int>> hv(nclass);
    std::vector<std::vector<System*>> cs(nclass);
    for (int r = 0; r < nsys; r++) {
        if (cls[r] < 0 || cls[r] >= nclass) fatal("batched classes: class index out of range");
        hv[cls[r]].push_back(handles[r]);
        cs[cls[r]].push_back(ss[r]);
    }
    std::vector<int> ctas(nclass), steps(nclass);
    long total = 0;
    for (int c = 0; c < nclass; c++) {
        ctas[c] = class_ctas[c];
        steps[c] = cs[c].empty() ? 0 : class_steps[c];
        if (steps[c] < 0) fatal("batched classes: negative step count");
        if (!cs[c].empty() && ctas[c] < (int)cs[c].size()) fatal("batched classes: fewer CTAs than systems in a class");
        if (!cs[c].empty()) total += ctas[c];
    }
    if (total > mixed_grid_blocks()) fatal("batched classes: more CTAs than SMs");
    batch_begin(ss, nclass);
    batch_run(hv, cs, ctas, steps);
    return batch_end(ss, handles, nclass);
}

// Choose the batched step's team partition exponent (CTAs per system ~ points^alpha)
// and the pair-force kernel's warp target by timing candidates on the listed systems:
// the field solves alone (their inputs are left unchanged; the MaZe unknown y is saved
// and restored) and the force stages alone (they only rewrite forces). Writes
// {alpha, warps, solve ms, forces ms} into out[0..3] and keeps the choice.
int mzb_batch_autotune(const int* handles, int nsys, double* out) {
    std::vector<System*> ss = batch_systems(handles, nsys);
    batch_begin(ss);
    Batch& B = g_batchst;
    cudaStream_t st = B.streams[0];
    const int nblocks = mixed_grid_blocks();
    MixedArgs* list_d = nullptr;
    int* start_d = nullptr;
    MZB_CHECK(cudaMalloc(&list_d, sizeof(MixedArgs) * nsys));
    MZB_CHECK(cudaMalloc(&start_d, sizeof(int) * (nsys + 1)));
    std::vector<double*> ysave(nsys, nullptr);
    MZB_CHECK(cudaDeviceSynchronize());  // the systems' streams have written y
    for (int r = 0; r < nsys; r++) {
        const int t = ss[r]->G.type;
        if (t == G_MAZE_LCG || t == G_MAZE_MG) {
            ysave[r] = dalloc<double>(ss[r]->G.m);
            copy_d2d(ysave[r], ss[r]->G.y, sizeof(double) * ss[r]->G.m);
        }
    }
    auto restore_y = [&]() {
        for (int r = 0; r < nsys; r++)
            if (ysave[r])
                MZB_CHECK(cudaMemcpyAsync(ss[r]->G.y, ysave[r], sizeof(double) * ss[r]->G.m, cudaMemcpyDeviceToDevice,
                                          st));
    };
    // One batched solve of every system's current charges from its previous field (the
    // work of an MD-step update; the solves write only the spare field buffer, the
    // multigrid levels and, restored here, the MaZe unknown), under the team partition of
    // exponent alpha; the mean of two timed launches after one untimed.
    auto time_set = [&](const std::vector<System*>& set, double alpha) {
        const int ns = (int)set.size();
        std::vector<MixedArgs> list(ns);
        size_t smem = 0;
        for (int r = 0; r < ns; r++) {
            double cst = 0.0;
            const int prog = mixed_update_prog(set[r]->G, cst);
            list[r] = mixed_args(*set[r], prog, cst);
            list[r].phi_old = set[r]->G.phi_prev();
            smem = std::max(smem, mixed_smem_bytes(list[r]));
        }
        upload(list_d, list.data(), sizeof(MixedArgs) * ns);
        const std::vector<int> start = team_starts(set, nblocks, alpha);
        upload(start_d, start.data(), sizeof(int) * (ns + 1));
        float tot = 0.f;
        for (int rep = 0; rep < 3; rep++) {
            restore_y();
            for (int r = 0; r < ns; r++) MZB_CHECK(cudaMemsetAsync(set[r]->bar, 0, sizeof(GridBarrier), st));
            MZB_CHECK(cudaEventRecord(B.t0, st));
            mixed_batch_launch(list_d, start_d, ns, nblocks, smem, st);
            MZB_CHECK(cudaEventRecord(B.t1, st));
            MZB_CHECK(cudaStreamSynchronize(st));
            float ms = 0.f;
            MZB_CHECK(cudaEventElapsedTime(&ms, B.t0, B.t1));
            if (rep > 0) tot += ms;
        }
        return (double)tot / 2;
    };
    auto time_solves = [&](double alpha) { return time_set(ss, alpha); };
    // team partition: CTAs per system ~ (grid points)^alpha
    const double alphas[] = {1.2, 1.0, 0.8, 0.6, 0.4};
    auto tune_alpha = [&](double& best_solve) {
        double best_alpha = B.alpha;
        best_solve = 1e30;
        for (double alpha : alphas) {
            const double ms = time_solves(alpha);
            if (ms < best_solve) {
                best_solve = ms;
                best_alpha = alpha;
            }
        }
        return best_alpha;
    };
    // Per size class (systems of one grid size), timed alone on all CTAs: the coarse-level
    // plan (each distinct one of mzb_set_mixed_plan; the FFT-solved coarse level pays off
    // with many CTAs per team, the levels down to 16^3 with few) and the time per grid
    // point of the fastest. The classes' shares of the mix are then weighted by that time
    // (the small grids' passes are latency-bound), so that the teams finish together, and
    // the exponent of the partition is tuned on the whole set.
    std::vector<int> sizes;
    for (System* s : ss)
        if (std::find(sizes.begin(), sizes.end(), s->G.n) == sizes.end()) sizes.push_back(s->G.n);
    std::vector<double> per_point(sizes.size(), 1.0);
    for (System* s : ss) s->G.batch_cost = 1.0;
    for (size_t c = 0; c < sizes.size(); c++) {
        std::vector<System*> cls;
        double pts = 0.0;
        for (System* s : ss)
            if (s->G.n == sizes[c]) {
                cls.push_back(s);
                pts += (double)s->G.m;
            }
        int best_plan = cls[0]->G.plan;
        double best_ms = 1e30;
        std::vector<std::pair<int, int>> seen;  // (levels, FFT coarse) of the plans timed
        for (int plan : {1, 2, 0}) {
            for (System* s : cls) {
                s->G.plan = plan;
                touch(*s);
                ensure_mixed_levels(s->G);
            }
            const std::pair<int, int> shape{cls[0]->G.nlev, cls[0]->G.coarse_fft ? 1 : 0};
            if (std::find(seen.begin(), seen.end(), shape) != seen.end()) continue;
            seen.push_back(shape);
            const double ms = time_set(cls, 1.0);
            if (ms < best_ms) {
                best_ms = ms;
                best_plan = plan;
            }
        }
        for (System* s : cls) {
            s->G.plan = best_plan;
            touch(*s);
            ensure_mixed_levels(s->G);
        }
        per_point[c] = best_ms / pts;
    }
    double ref = per_point[0];
    for (double v : per_point) ref = std::min(ref, v);
    for (System* s : ss)
        for (size_t c = 0; c < sizes.size(); c++)
            if (s->G.n == sizes[c]) s->G.batch_cost = per_point[c] / ref;
    double best_solve = 0.0;
    B.alpha = tune_alpha(best_solve);
    restore_y();
    MZB_CHECK(cudaStreamSynchronize(st));
    for (double* p : ysave)
        if (p) cudaFree(p);
    cudaFree(list_d);
    cudaFree(start_d);

    // pair forces of all systems together (their work division is fixed by N; timed only)
    double best_forces = 0.0;
    long force_ctas = 0;
    for (System* s : ss) force_ctas += s->P.tf_nst;
    {
        float tot = 0.f;
        for (int rep = 0; rep < 3; rep++) {
            MZB_CHECK(cudaEventRecord(B.t0, st));
            MZB_CHECK(cudaEventRecord(B.fork1, st));
            for (int r = 0; r < nsys; r++) {
                MZB_CHECK(cudaStreamWaitEvent(ss[r]->stream, B.fork1, 0));
                build_cells(ss[r]->P, ss[r]->stream);
                tf_forces(ss[r]->P, ss[r]->stream);
                MZB_CHECK(cudaEventRecord(B.join1[r], ss[r]->stream));
                MZB_CHECK(cudaStreamWaitEvent(st, B.join1[r], 0));
            }
            MZB_CHECK(cudaEventRecord(B.t1, st));
            MZB_CHECK(cudaStreamSynchronize(st));
            float ms = 0.f;
            MZB_CHECK(cudaEventElapsedTime(&ms, B.t0, B.t1));
            if (rep > 0) tot += ms;
        }
        best_forces = tot / 2;
    }
    for (System* s : ss) touch(*s);
    batch_clear_graphs();
    if (out) {
        out[0] = B.alpha;
        out[1] = (double)force_ctas;
        out[2] = best_solve;
        out[3] = best_forces;
    }
    return 0;
}

// Bytes of device memory one system of n^3 grid points and n_p ions holds with the
// FP32+refine field solve (fields, multigrid levels, the resident kernels' work area, particle
// and pair-force arrays);
// the request loop admits jobs against an HBM budget with it.
double mzb_system_footprint(int n, int n_p) {
    const double m = (double)n * n * n;
    double levels = 0.0;
    int sizes[kMixedMaxLevels];
    const int L = mixed_levels(n, sizes);
    for (int l = 0; l < L; l++) levels += 3.0 * 4.0 * (double)sizes[l] * sizes[l] * sizes[l];
    levels += 8.0 * (double)(n / 2) * (n / 2) * (n / 4 + 1);  // half spectrum of an FFT-solved coarse level
    const double grid = 8.0 * m * 10.0;  // q, phi x3, y, r, p0, p1, Ap, tmp
    const TfShape t = tf_shape(n_p);
    const double super_tiles = 0.5 * t.nsb * (t.nsb + 1.0);  // pair-force CTAs
    // per ion: seven vectors, the lists, the spline weights (whether or not the scheme has them);
    // per super-tile: force partials, gather entries, energy
    const double parts = (double)n_p * (8.0 * 3 * 7 + 4.0 * 8 + 8.0 * 12) +
                         super_tiles * (2.0 * t.sb * (32 * 3 * 8.0 + 4.0) + 16.0);
    const double halo = (double)resident_halo_bytes(n);  // the bootstrap's FP64 solve
    return grid + levels + parts + halo + 64.0 * 1024 * 1024;
}

}  // extern "C"

// ====================================================================================
// Output snapshots (this build's extension). The reference's output path calls the
// synchronous getters every `stride` steps (maze_poisson/myio/output/csv.py:45-183,
// solver.py:461-464). A snapshot instead stages the requested arrays with
// device-to-device copies on the system's stream (ordered after the last step and before
// the next one), then copies the staging area to pinned host memory on a separate copy
// stream, so the transfer overlaps the following MD steps. Two slots per system.
// ====================================================================================
namespace mzb {
namespace {

enum SnapBits { SNAP_POS = 1, SNAP_VEL = 2, SNAP_FORCES = 4, SNAP_SCALARS = 8, SNAP_FIELDS = 16 };

struct SnapSlot {
    int what = 0;
    bool busy = false;
    long np = 0, m = 0;
    cudaEvent_t staged = nullptr, done = nullptr;
    double* d_buf = nullptr;
    double* h_buf = nullptr;
    size_t cap = 0;  // doubles
};

struct SnapState {
    cudaStream_t copy = nullptr;
    SnapSlot slot[2];
};

std::vector<SnapState*> g_snaps;  // per system handle

SnapState& snap_state() {
    if (g_current < 0) fatal("no system selected");
    if ((int)g_snaps.size() <= g_current) g_snaps.resize(g_current + 1, nullptr);
    SnapState*& st = g_snaps[g_current];
    if (!st) {
        st = new SnapState();
        MZB_CHECK(cudaStreamCreateWithFlags(&st->copy, cudaStreamNonBlocking));
        for (auto& sl : st->slot) {
            MZB_CHECK(cudaEventCreateWithFlags(&sl.staged, cudaEventDisableTiming));
            MZB_CHECK(cudaEventCreateWithFlags(&sl.done, cudaEventDisableTiming));
        }
    }
    return *st;
}

// Layout of a slot's buffer: pos, vel (np*3 each), fcs_elec, fcs_noel, fcs_tot (np*3
// each), scalars (8: q total, V_notelec, K, Px, Py, Pz, T, spare), phi, phi_prev (m each).
size_t snap_size(long np, long m, int what) {
    size_t s = 5 * 3 * (size_t)np + 8;
    if (what & SNAP_FIELDS) s += 2 * (size_t)m;
    return s;
}

}  // namespace

namespace {
void release_snapshots(int handle) {
    if (handle < 0 || handle >= (int)g_snaps.size() || !g_snaps[handle]) return;
    SnapState* st = g_snaps[handle];
    cudaStreamSynchronize(st->copy);
    for (auto& sl : st->slot) {
        if (sl.d_buf) cudaFree(sl.d_buf);
        if (sl.h_buf) cudaFreeHost(sl.h_buf);
        cudaEventDestroy(sl.staged);
        cudaEventDestroy(sl.done);
    }
    cudaStreamDestroy(st->copy);
    delete st;
    g_snaps[handle] = nullptr;
}
}  // namespace
}  // namespace mzb

extern "C" {

// Queue a snapshot of the selected system (what: 1 positions, 2 velocities, 4 forces
// (elec, noel, tot), 8 scalars (V_notelec, K, momentum, T), 16 fields (phi, phi_prev)).
// Returns the slot (0 or 1) to fetch, or -1 if both slots hold unfetched snapshots.
int mzb_snapshot_begin(int what) {
    System& s = sys();
    ParticleDev& P = parts();
    SnapState& st = snap_state();
    int k = !st.slot[0].busy ? 0 : (!st.slot[1].busy ? 1 : -1);
    if (k < 0) return -1;
    SnapSlot& sl = st.slot[k];
    const bool fields = (what & SNAP_FIELDS) && s.G.ready;
    const long m = fields ? s.G.m : 0;
    const size_t need = snap_size(P.np, m, fields ? what : what & ~SNAP_FIELDS);
    if (need > sl.cap) {
        if (sl.d_buf) cudaFree(sl.d_buf);
        if (sl.h_buf) cudaFreeHost(sl.h_buf);
        MZB_CHECK(cudaMalloc(&sl.d_buf, need * sizeof(double)));
        MZB_CHECK(cudaMallocHost(&sl.h_buf, need * sizeof(double)));
        sl.cap = need;
    }
    sl.what = fields ? what : what & ~SNAP_FIELDS;
    sl.np = P.np;
    sl.m = m;
    const size_t v = 3 * (size_t)P.np * sizeof(double);
    double* d = sl.d_buf;
    if (what & SNAP_SCALARS) kinetic_and_momentum(P, s.stream);
    if (P.np > 0) {
        if (what & SNAP_POS) MZB_CHECK(cudaMemcpyAsync(d, P.pos, v, cudaMemcpyDeviceToDevice, s.stream));
        if (what & SNAP_VEL) MZB_CHECK(cudaMemcpyAsync(d + 3 * P.np, P.vel, v, cudaMemcpyDeviceToDevice, s.stream));
        if (what & SNAP_FORCES) {
            MZB_CHECK(cudaMemcpyAsync(d + 6 * P.np, P.fe, v, cudaMemcpyDeviceToDevice, s.stream));
            MZB_CHECK(cudaMemcpyAsync(d + 9 * P.np, P.fn, v, cudaMemcpyDeviceToDevice, s.stream));
            MZB_CHECK(cudaMemcpyAsync(d + 12 * P.np, P.ft, v, cudaMemcpyDeviceToDevice, s.stream));
        }
    }
    if (what & SNAP_SCALARS)
        MZB_CHECK(cudaMemcpyAsync(d + 15 * P.np, P.red, 8 * sizeof(double), cudaMemcpyDeviceToDevice, s.stream));
    if (fields) {
        double* f = d + 15 * P.np + 8;
        MZB_CHECK(cudaMemcpyAsync(f, s.G.phi(), sizeof(double) * m, cudaMemcpyDeviceToDevice, s.stream));
        if (s.G.type != G_FFT)
            MZB_CHECK(cudaMemcpyAsync(f + m, s.G.phi_prev(), sizeof(double) * m, cudaMemcpyDeviceToDevice, s.stream));
    }
    MZB_CHECK(cudaEventRecord(sl.staged, s.stream));
    MZB_CHECK(cudaStreamWaitEvent(st.copy, sl.staged, 0));
    MZB_CHECK(cudaMemcpyAsync(sl.h_buf, sl.d_buf, need * sizeof(double), cudaMemcpyDeviceToHost, st.copy));
    MZB_CHECK(cudaEventRecord(sl.done, st.copy));
    sl.busy = true;
    return k;
}

// Wait for snapshot `slot` of the selected system and return its pinned host buffer
// (read in place, no copy): pos, vel, fcs_elec, fcs_noel, fcs_tot (n_p*3 doubles each),
// 8 scalars, then phi and phi_prev (n^3 each) if captured. The buffer stays valid until
// the slot is released by mzb_snapshot_fetch. Null if the slot holds no snapshot.
double* mzb_snapshot_host(int slot) {
    if (slot < 0 || slot > 1) return nullptr;
    SnapState& st = snap_state();
    SnapSlot& sl = st.slot[slot];
    if (!sl.busy) return nullptr;
    MZB_CHECK(cudaEventSynchronize(sl.done));
    return sl.h_buf;
}

// Wait for snapshot `slot` of the selected system and copy it out; null pointers skip an
// array. scalars[8] = {q total, V_notelec, K, Px, Py, Pz, T, 0}. Returns the mask that
// was captured, or -1 if the slot holds no snapshot.
int mzb_snapshot_fetch(int slot, double* pos, double* vel, double* fcs_elec, double* fcs_noel, double* fcs_tot,
                       double* scalars, double* phi, double* phi_prev) {
    if (slot < 0 || slot > 1) return -1;
    SnapState& st = snap_state();
    SnapSlot& sl = st.slot[slot];
    if (!sl.busy) return -1;
    MZB_CHECK(cudaEventSynchronize(sl.done));
    const size_t v = 3 * (size_t)sl.np * sizeof(double);
    const double* h = sl.h_buf;
    if ((sl.what & SNAP_POS) && pos) memcpy(pos, h, v);
    if ((sl.what & SNAP_VEL) && vel) memcpy(vel, h + 3 * sl.np, v);
    if (sl.what & SNAP_FORCES) {
        if (fcs_elec) memcpy(fcs_elec, h + 6 * sl.np, v);
        if (fcs_noel) memcpy(fcs_noel, h + 9 * sl.np, v);
        if (fcs_tot) memcpy(fcs_tot, h + 12 * sl.np, v);
    }
    if ((sl.what & SNAP_SCALARS) && scalars) {
        memcpy(scalars, h + 15 * sl.np, 8 * sizeof(double));
        scalars[7] = 0.0;
    }
    if (sl.what & SNAP_FIELDS) {
        if (phi) memcpy(phi, h + 15 * sl.np + 8, sizeof(double) * sl.m);
        if (phi_prev) memcpy(phi_prev, h + 15 * sl.np + 8 + sl.m, sizeof(double) * sl.m);
    }
    sl.busy = false;
    return sl.what;
}

}  // extern "C"
