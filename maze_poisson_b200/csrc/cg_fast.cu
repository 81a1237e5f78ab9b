// FP64 conjugate-gradient field solves with a TMA-staged 2.5-D stencil (sm_100a).
//
// Serves the CG programs of the solver engine -- conj_grad (library/src/plcg.c:28-90),
// its explicit-Jacobi form (plcg.c:104-166 with precond_jacobi.c:8-14), the LCG field
// init/update (grid_lcg.c:100-149) and the MaZe constraint solve (verlet.c:31-71) -- for
// grids with n % 16 == 0 and 16 <= n <= 256. Arithmetic per point is the reference's
// (same operation order, every product rounded), so single sweeps match bit for bit;
// only the dot products are summed in a different (fixed) order.
//
// One persistent CTA per SM (cooperative launch): 31 warps compute, one issues the TMA loads.
// The grid is cut into nj x ni blocks of planes x rows, one per CTA (cg_fast_plan), the same
// points in every phase. Per CG iteration:
//   phase A: p <- beta p + z(r), Ap = L p, <p, Ap>. The CTA marches up the planes: (rows+2) x n
//     slabs of p_old and r arrive by TMA (one bulk-tensor copy per array, j wrapped) into a
//     ring; each thread turns its column pair into p_new once, keeps p_new(i-1), p_new(i),
//     p_new(i+1) in registers and reads the j+-1 / k+-1 neighbours from a shared p_new plane.
//   grid reduction, alpha = <r, z> / <p, Ap>; phase B's first slabs are fetched meanwhile
//   phase B: r += alpha Ap, <r, r>, max |r|, down the planes; in every second iteration also x,
//     for the two directions it lacks: the two ping-pong p grids are both there, the sums are
//     added in the same order, and x costs 4 grid passes in 2 iterations instead of 6.
//   grid reduction, convergence test, beta. A direction that x still lacks is added at the end.
//
// Cost. An iteration passes 9 grids through memory (A: 2 in, 2 out; B: 2 in, 1 out, and every
// second time 3 in, 1 out more), 187 us at 256^3 at the copy bandwidth of 6.45 TB/s. Measured us
// per iteration, n = 160 / 192 / 240 / 256: 89 / 133 / 228 / 270 before, 59 / 96 / 180 / 202 now
// (256: A 90, B 53 and 125, reductions 9 and 12). What it took, at 256: blocks that march in
// step, x every second iteration and phase B through a bulk-copy ring 270 -> 240; no read of
// the global timer ahead of a wait 240 -> 220; a warp of its own for issuing loads, which took
// 0.6 us a slab in a computing warp that all others then waited for, 220 -> 202. 1024 threads of
// one pair beat 512 of two. Phase B upwards instead of downwards: 15 % slower.
#include <cudaTypedefs.h>

#include <algorithm>

#include "engine.cuh"
#include "tma.cuh"

namespace mzb {

struct CgFastArgs {
    int prog;   // PROG_CG, PROG_INIT_FIELD, PROG_LCG_UPDATE, PROG_MAZE_LCG
    int kind;   // PC_IMPLICIT or PC_JACOBI
    int n, stages;
    int rows, nj, ni;  // blocks of at most `rows` rows: nj along j, ni along i, one per CTA
    double tol, c;
    const double* q;
    const double* phi_old;
    const double* phi_prev;
    double* phi_new;
    double* y;
    const double* b;
    const double* x0;
    double* x;
    double* r;
    double* p0;
    double* p1;
    double* Ap;
    double* tmp;
    double* partials;
    GridBarrier* bar;
    int* result;
    unsigned long long* stamps;  // optional phase timestamps (block 0), see stamp()
};

namespace {

constexpr int kThreads = 1024;
constexpr int kProducer = kThreads - 32;  // the last warp issues the TMA loads, the others compute
constexpr int kMaxStages = 6;

// The CTA's points: planes [i0, i1), rows [j0, j1).
struct Block {
    int i0, i1, j0, j1;
};
__device__ __forceinline__ Block block_of(const CgFastArgs& a) {
    const int jb = blockIdx.x % a.nj, ib = blockIdx.x / a.nj;
    return Block{ib * a.n / a.ni, (ib + 1) * a.n / a.ni, jb * a.n / a.nj, (jb + 1) * a.n / a.nj};
}

struct Nbr {
    long c, ip, im, jp, jm, kp, km;
};
__device__ __forceinline__ Nbr nbr_of(int n, int i, int j, int k) {
    const long n2 = (long)n * n;
    Nbr o;
    o.c = ((long)i * n + j) * n + k;
    o.ip = o.c + (i + 1 == n ? -(long)(n - 1) * n2 : n2);
    o.im = o.c + (i == 0 ? (long)(n - 1) * n2 : -n2);
    o.jp = o.c + (j + 1 == n ? -(long)(n - 1) * n : (long)n);
    o.jm = o.c + (j == 0 ? (long)(n - 1) * n : -(long)n);
    o.kp = o.c + (k + 1 == n ? -(long)(n - 1) : 1L);
    o.km = o.c + (k == 0 ? (long)(n - 1) : -1L);
    return o;
}
template <class F>
__device__ __forceinline__ double lap7(const Nbr& o, F&& f) {
    double s = f(o.ip) + f(o.im);
    s = s + f(o.jp);
    s = s + f(o.jm);
    s = s + f(o.kp);
    s = s + f(o.km);
    return s - f(o.c) * 6.0;
}

// Visit the CTA's own points.
template <class F>
__device__ __forceinline__ void for_own(const CgFastArgs& a, const Block& w, F&& f) {
    const int n = a.n, per = (w.j1 - w.j0) * n;
    for (int i = w.i0; i < w.i1; i++)
        for (int c = threadIdx.x; c < per; c += kThreads) f(i, w.j0 + c / n, c % n);
}

// NS sums then NM maxima over the grid; deterministic fixed-order gather.
template <int NS, int NM>
__device__ bool reduce(double* s, double* mx, const CgFastArgs& a, unsigned& epoch, int& seq) {
    __shared__ double sh[4 * 32];
    __shared__ double res[4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const long G = gridDim.x;
#pragma unroll
    for (int q = 0; q < NS; q++) s[q] = warp_sum(s[q]);
#pragma unroll
    for (int q = 0; q < NM; q++) mx[q] = warp_max(mx[q]);
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NS; q++) sh[q * 32 + w] = s[q];
#pragma unroll
        for (int q = 0; q < NM; q++) sh[(NS + q) * 32 + w] = mx[q];
    }
    __syncthreads();
    double* part = a.partials + (long)(seq & 1) * 4 * G;
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < NS + NM; q++) {
            double v = lane < nwarp ? sh[q * 32 + lane] : 0.0;
            v = q < NS ? warp_sum(v) : warp_max(v);
            if (lane == 0) part[q * G + blockIdx.x] = v;
        }
    }
    const bool ok = grid_sync_mono(a.bar, epoch);
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < NS + NM; q++) {
            double v = 0.0;
            for (long b = lane; b < G; b += 32) {
                const double e = __ldcg(part + q * G + b);
                v = q < NS ? v + e : fmax(v, e);
            }
            v = q < NS ? warp_sum(v) : warp_max(v);
            if (lane == 0) res[q] = v;
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NS; q++) s[q] = res[q];
#pragma unroll
    for (int q = 0; q < NM; q++) mx[q] = res[NS + q];
    __syncthreads();
    seq++;
    return ok;
}

// slots 0..3: set-up; 4 + 4 it + {0..3}: phase ends of iteration it < kCgStampIters;
// 40 + 2 e + {0, 1}: slab e of the first phase A (compute done, next stage landed)
__device__ __forceinline__ void stamp(const CgFastArgs& a, int slot) {
    if (a.stamps != nullptr && blockIdx.x == 0 && threadIdx.x == 0 && slot < 96)
        a.stamps[slot] = global_ns();
}
__device__ __forceinline__ void stamp_it(const CgFastArgs& a, long iter, int k) {
    if (iter < kCgStampIters) stamp(a, 4 + 4 * (int)iter + k);
}

// z(r): the direction increment of the preconditioned residual, exactly as the
// reference forms it: (1/6) r (conj_grad, plcg.c:342-343,369-370) or
// -1 * (-r / 6) (conj_grad_precond with the Jacobi preconditioner).
template <int KIND>
__device__ __forceinline__ double zf(double r) {
    if (KIND == PC_IMPLICIT) return (1.0 / 6.0) * r;
    return -1.0 * (-r / 6.0);
}


// Ring of phase B: plane slabs (contiguous in the grid) of r and Ap (kDepth2 deep) or of r,
// Ap, x and two directions (kDepth5 deep), in the shared memory that phase A's stages and
// planes take otherwise (cg_fast_plan sees to it that it fits).
constexpr int kDepth2 = 5, kDepth5 = 2;
struct UpdateRing {
    uint64_t* full;
    uint64_t* empty;
    double* buf;
    int used, issued;  // slabs that have gone through it, and issued (thread kProducer), in this launch
};

// evict_first for what is read for the last time (Ap, x, the older p): 5 % at 144^3, nothing at 256^3
__device__ __forceinline__ void bulk_load_ef(double* dst, const double* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_first.b64 pol, 1.0;\n\t"
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], pol;\n\t}" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void bulk_load(double* dst, const double* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Issue slab e of phase B (plane i1 - 1 - e). One thread.
template <int NA>
__device__ __forceinline__ void update_issue(const CgFastArgs& a, UpdateRing& q, const Block& own, int e, const double* X,
                                             const double* p0, const double* p1) {
    constexpr int D = NA == 2 ? kDepth2 : kDepth5;
    const int n = a.n, size = (own.j1 - own.j0) * n, s = (q.used + e) % D;
    const long o = ((long)(own.i1 - 1 - e) * n + own.j0) * n;
    const uint32_t bytes = (uint32_t)(size * sizeof(double));
    double* dst = q.buf + s * NA * size;
    mbar_expect_tx(&q.full[s], NA * bytes);
    q.issued++;
    bulk_load(dst, a.r + o, bytes, &q.full[s]);
    bulk_load_ef(dst + size, a.Ap + o, bytes, &q.full[s]);
    if (NA == 5) {
        bulk_load_ef(dst + 2 * size, X + o, bytes, &q.full[s]);
        bulk_load_ef(dst + 3 * size, p0 + o, bytes, &q.full[s]);
        bulk_load(dst + 4 * size, p1 + o, bytes, &q.full[s]);
    }
}

// Phase B over the CTA's own points: r += alpha Ap, <r, r> (and <r, P r> for Jacobi), max |r|;
// NA = 5: x += alpha0 p0, then x += alpha p1. The first slabs were issued before the reduction
// that yields alpha. A copy that does not land sets *abort_sh.
template <int KIND, int NA>
__device__ __forceinline__ void update_own(const CgFastArgs& a, UpdateRing& q, const Block& own, double* X,
                                           const double* p0, double alpha0, const double* p1, double alpha,
                                           double* sums, double* rmax, int* abort_sh) {
    constexpr int D = NA == 2 ? kDepth2 : kDepth5;
    const int n = a.n, size = (own.j1 - own.j0) * n, count = own.i1 - own.i0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, v = 2 * (int)threadIdx.x;
    long o = ((long)(own.i1 - 1) * n + own.j0) * n + v;
    if (warp == kProducer / 32) {
        if (lane == 0)
            for (int e = D; e < count && !*abort_sh; e++) {
                const int sq = q.used + e - D;  // the slab that leaves the stage
                if (mbar_wait(&q.empty[sq % D], (uint32_t)((sq / D) & 1)))
                    update_issue<NA>(a, q, own, e, X, p0, p1);
                else
                    *abort_sh = 1;
            }
        __syncwarp();
        q.used += count;
        return;
    }
    for (int e = 0; e < count; e++) {
        const int sq = q.used + e, s = sq % D;
        int good = 1;
        if (lane == 0 && (*abort_sh || !mbar_wait(&q.full[s], (uint32_t)((sq / D) & 1)))) good = 0;
        good = __shfl_sync(0xffffffffu, good, 0);
        if (!good) *abort_sh = 1;
        if (good && v < size) {
            const double* b = q.buf + s * NA * size + v;
            double2 rr = *reinterpret_cast<const double2*>(b);
            const double2 aa = *reinterpret_cast<const double2*>(b + size);
            rr.x = rr.x + alpha * aa.x;
            rr.y = rr.y + alpha * aa.y;
            *reinterpret_cast<double2*>(a.r + o) = rr;
            if (NA == 5) {
                double2 xx = *reinterpret_cast<const double2*>(b + 2 * size);
                const double2 pa = *reinterpret_cast<const double2*>(b + 3 * size);
                const double2 pb = *reinterpret_cast<const double2*>(b + 4 * size);
                xx.x = xx.x + alpha0 * pa.x;
                xx.y = xx.y + alpha0 * pa.y;
                xx.x = xx.x + alpha * pb.x;
                xx.y = xx.y + alpha * pb.y;
                __stcs(reinterpret_cast<double2*>(X + o), xx);
            }
            sums[0] += rr.x * rr.x;
            sums[0] += rr.y * rr.y;
            if (KIND == PC_JACOBI) {
                sums[1] += rr.x * (-rr.x / 6.0);
                sums[1] += rr.y * (-rr.y / 6.0);
            }
            rmax[0] = fmax(rmax[0], fmax(fabs(rr.x), fabs(rr.y)));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&q.empty[s]);
        o -= (long)n * n;
    }
    q.used += count;
}

template <int KIND>  // PrecondKind
__global__ void __launch_bounds__(kThreads, 1)
    cg_fast_kernel(const __grid_constant__ CUtensorMap map_r_row, const __grid_constant__ CUtensorMap map_r_slab,
                   const __grid_constant__ CUtensorMap map_p0_row, const __grid_constant__ CUtensorMap map_p0_slab,
                   const __grid_constant__ CUtensorMap map_p1_row, const __grid_constant__ CUtensorMap map_p1_slab,
                   CgFastArgs a) {
    extern __shared__ __align__(128) unsigned char smraw[];
    const int n = a.n, R = a.rows + 2, S = a.stages;
    const int slab = R * n;  // doubles per array per stage
    const Block own = block_of(a);
    const int rows = own.j1 - own.j0, nload = own.i1 - own.i0 + 2;
    // TMA destinations must start on 128-byte boundaries of the shared window
    unsigned char* sm0 = smraw + ((128u - (smem_u32(smraw) & 127u)) & 127u);
    double* stg = reinterpret_cast<double*>(sm0);  // [S][2][R][n]: p_old, r slabs
    double* pnb = stg + S * 2 * slab;        // [2][R][n]: p_new planes
    double* wrp = pnb + 2 * slab;                  // [S][2][n]: the wrapped halo row, if the block has one
    uint64_t* full = reinterpret_cast<uint64_t*>(wrp + S * 2 * n);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (a.prog != PROG_CG && a.prog != PROG_INIT_FIELD && a.prog != PROG_LCG_UPDATE &&
        a.prog != PROG_MAZE_LCG) {
        if (blockIdx.x == 0 && tid == 0) {
            a.result[0] = -1;
            a.result[1] = 2;
        }
        return;
    }
    __shared__ int abort_sh;
    __shared__ __align__(8) uint64_t ubar[2 * (kDepth2 + kDepth5)];
    UpdateRing q2{ubar, ubar + kDepth2, stg, 0, 0}, q5{ubar + 2 * kDepth2, ubar + 2 * kDepth2 + kDepth5, stg, 0, 0};
    if (tid == 0) {
        for (int s = 0; s < S; s++) mbar_init(&full[s], 1);
        for (int s = 0; s < kDepth2; s++) {
            mbar_init(&q2.full[s], 1);
            mbar_init(&q2.empty[s], kProducer / 32);
        }
        for (int s = 0; s < kDepth5; s++) {
            mbar_init(&q5.full[s], 1);
            mbar_init(&q5.empty[s], kProducer / 32);
        }
        fence_mbar_init();
        abort_sh = 0;
    }
    if (tid == kProducer) {
        prefetch_tensormap(&map_r_row); prefetch_tensormap(&map_r_slab);
        prefetch_tensormap(&map_p0_row); prefetch_tensormap(&map_p0_slab);
        prefetch_tensormap(&map_p1_row); prefetch_tensormap(&map_p1_slab);
    }
    __syncthreads();

    unsigned epoch = 0;
    int seq = 0;
    bool ok = true;
    int result = -1;

    // ---- set-up of the right-hand side (one pass over own points) ----
    if (a.prog == PROG_INIT_FIELD) {        // y = 0; phi = c q   (grid_lcg.c:108-113)
        for_own(a, own, [&](int i, int j, int k) {
            const long c = ((long)i * n + j) * n + k;
            a.y[c] = 0.0;
            a.phi_new[c] = a.q[c] * a.c;
        });
    } else if (a.prog == PROG_LCG_UPDATE) { // y = c q            (grid_lcg.c:134-138)
        for_own(a, own, [&](int i, int j, int k) {
            const long c = ((long)i * n + j) * n + k;
            a.y[c] = a.q[c] * a.c;
        });
    } else if (a.prog == PROG_MAZE_LCG) {   // phi = 2 phi - phi_prev; sigma = L phi + c q
        for_own(a, own, [&](int i, int j, int k) {
            const Nbr o = nbr_of(n, i, j, k);
            auto ex = [&](long q) { return 2 * a.phi_old[q] - a.phi_prev[q]; };
            a.phi_new[o.c] = ex(o.c);
            a.tmp[o.c] = lap7(o, ex) + a.c * a.q[o.c];
        });
    }
    stamp(a, 0);
    ok = grid_sync_mono(a.bar, epoch);
    stamp(a, 1);
    const double* B = a.prog == PROG_INIT_FIELD ? a.phi_new
                      : a.prog == PROG_LCG_UPDATE ? a.y
                      : a.prog == PROG_MAZE_LCG ? a.tmp : a.b;
    const double* X0 = a.prog == PROG_INIT_FIELD ? a.y
                       : a.prog == PROG_LCG_UPDATE ? a.phi_old
                       : a.prog == PROG_MAZE_LCG ? a.y : a.x0;
    double* X = (a.prog == PROG_INIT_FIELD || a.prog == PROG_LCG_UPDATE) ? a.phi_new
                : a.prog == PROG_MAZE_LCG ? a.y : a.x;

    // ---- r = L x0 - b; x = x0; <r, z(r)> ----
    double rv = 0.0;
    if (ok) {
        double acc[1] = {0.0}, m0[1];
        for_own(a, own, [&](int i, int j, int k) {
            const Nbr o = nbr_of(n, i, j, k);
            const double x0c = X0[o.c];
            const double rr = lap7(o, [&](long q) { return X0[q]; }) + -1.0 * B[o.c];
            if (X != X0) X[o.c] = x0c;
            a.r[o.c] = rr;
            acc[0] += rr * (KIND == PC_IMPLICIT ? rr * (1.0 / 6.0) : -rr / 6.0);
        });
        ok = reduce<1, 0>(acc, m0, a, epoch, seq);
        rv = KIND == PC_IMPLICIT ? -acc[0] : acc[0];
    }
    stamp(a, 2);

    // phase A streams planes i0 - 1 .. i1 (wrapped)
    const bool lo = own.j0 == 0, hi = own.j1 == n;  // at most one (nj >= 2)
    const uint32_t stage_bytes = (uint32_t)((2 * slab + (lo || hi ? 2 * n : 0)) * sizeof(double));

    // the thread's column pair (k, k+1) of the slab, if it has one
    const bool pv = tid < rows * n / 2;
    const int go = pv ? 2 * tid : 0, k = go % n;  // offset in the slab
    const int so = go + n;                        // in the stage and the plane
    // halo pairs of the p_new plane: rows 0 and rows + 1, n/2 pairs each, by the last threads
    const int ht = tid - (kProducer - n);
    const bool hv = ht >= 0 && ht < n;
    const int hrow = ht < n / 2 ? 0 : rows + 1, hk = hv ? 2 * (ht % (n / 2)) : 0;
    const bool wrapped = hrow == 0 ? lo : hi;
    // Issue slab e of phase A into stage s. All of the producer warp.
    auto issue = [&](int e, int s, const CUtensorMap* mslab, const CUtensorMap* mrow) {
        int plane = own.i0 - 1 + e;
        plane += plane < 0 ? n : plane >= n ? -n : 0;
        if (lane == 0) mbar_expect_tx(&full[s], stage_bytes);
        __syncwarp();
        // one (n x R) box per array from row j0-1 (rows outside [0,n) are zero-filled);
        // the periodic image of a wrapped row goes to the wrap buffer
        if (lane < 2) tma_load_3d(stg + (2 * s + lane) * slab, lane ? &map_r_slab : mslab, 0, own.j0 - 1, plane, &full[s]);
        if ((lo || hi) && lane >= 2 && lane < 4)
            tma_load_3d(wrp + (2 * s + lane - 2) * n, lane == 3 ? &map_r_row : mrow, 0, lo ? n - 1 : 0, plane, &full[s]);
    };

    const long limit = (long)n * n;
    long iter = 0;
    int ld = 0;  // slabs of phase A issued so far (producer warp)
    int cs = 0;  // stage and parity of the next one
    uint32_t cph = 0;
    double beta = 0.0;
    const double* pold = a.p1;
    double* pnew = a.p0;
    const double* pend = nullptr;  // direction x still lacks, and its alpha
    double apend = 0.0;
    while (ok && iter < limit) {
        const bool first = iter == 0;
        const CUtensorMap* mslab = (pold == a.p0) ? &map_p0_slab : &map_p1_slab;
        const CUtensorMap* mrow = (pold == a.p0) ? &map_p0_row : &map_p1_row;
        double pap[1] = {0.0}, m0[1];
        if (tid >= kProducer) {
            fence_proxy_async_global();
            for (int e = 0; e < nload && e < S - 1; e++, ld++) issue(e, (cs + e) % S, mslab, mrow);
        }
        double2 pprev = make_double2(0.0, 0.0), pcur = pprev, pnext = pprev;
        int buf = 0;
        for (int e = 0; e < nload; e++) {
            const int s = cs;
            // the stage of the slab before is free: every warp has passed the barrier after it
            if (tid >= kProducer && e + S - 1 < nload && !abort_sh) {
                issue(e + S - 1, s == 0 ? S - 1 : s - 1, mslab, mrow);
                ld++;
            }
            int good = 1;
            if (lane == 0 && tid < kProducer && (abort_sh || !mbar_wait(&full[s], cph))) good = 0;
            good = __shfl_sync(0xffffffffu, good, 0);
            if (!good) abort_sh = 1;
            if (first && e < 18 && tid == 0) stamp(a, 40 + 3 * e);
            const double* sp = stg + 2 * s * slab;  // p_old rows
            const double* sr = sp + slab;           // r rows
            const bool fill = e > 0 && e + 1 < nload;
            double* pb = pnb + buf * slab;
            if (good) {
                // this slab's p_new on the own pair (and, for planes ia..ib, the shared plane)
                if (pv) {
                    const double2 rr = *reinterpret_cast<const double2*>(sr + so);
                    double2 z = make_double2(zf<KIND>(rr.x), zf<KIND>(rr.y));
                    if (!first) {
                        const double2 po = *reinterpret_cast<const double2*>(sp + so);
                        z.x = po.x * beta + z.x;
                        z.y = po.y * beta + z.y;
                    }
                    pnext = z;
                    if (fill) *reinterpret_cast<double2*>(pb + so) = z;
                }
                if (fill && hv) {
                    const double* hp = wrapped ? wrp + 2 * s * n : sp + hrow * n;
                    const double* hr = hp + (wrapped ? n : slab);
                    const double2 rr = *reinterpret_cast<const double2*>(hr + hk);
                    double2 z = make_double2(zf<KIND>(rr.x), zf<KIND>(rr.y));
                    if (!first) {
                        const double2 po = *reinterpret_cast<const double2*>(hp + hk);
                        z.x = po.x * beta + z.x;
                        z.y = po.y * beta + z.y;
                    }
                    *reinterpret_cast<double2*>(pb + hrow * n + hk) = z;
                }
            }
            if (first && e < 18 && tid == 0) stamp(a, 41 + 3 * e);
            if (e >= 2 && good && pv) {
                // output plane i0 + e - 2; its p_new plane is in the other buffer
                const double* pc = pnb + (buf ^ 1) * slab;
                const double2 jp = *reinterpret_cast<const double2*>(pc + so + n);
                const double2 jm = *reinterpret_cast<const double2*>(pc + so - n);
                const double km = pc[k == 0 ? so + n - 1 : so - 1];
                const double kp2 = pc[k + 2 == n ? so + 2 - n : so + 2];
                double s0 = pnext.x + pprev.x;
                s0 = s0 + jp.x;
                s0 = s0 + jm.x;
                s0 = s0 + pcur.y;
                s0 = s0 + km;
                double s1 = pnext.y + pprev.y;
                s1 = s1 + jp.y;
                s1 = s1 + jm.y;
                s1 = s1 + kp2;
                s1 = s1 + pcur.x;
                const double2 ap = make_double2(s0 - pcur.x * 6.0, s1 - pcur.y * 6.0);
                const long g = ((long)(own.i0 + e - 2) * n + own.j0) * n + go;
                *reinterpret_cast<double2*>(pnew + g) = pcur;
                *reinterpret_cast<double2*>(a.Ap + g) = ap;
                pap[0] += pcur.x * ap.x;
                pap[0] += pcur.y * ap.y;
            }
            if (first && e < 18 && tid == 0) stamp(a, 42 + 3 * e);
            __syncthreads();  // p_new planes complete / free again, stage s too
            pprev = pcur;
            pcur = pnext;
            if (fill) buf ^= 1;
            if (++cs == S) {
                cs = 0;
                cph ^= 1;
            }
        }
        // the CTA's own writes of this phase are read by bulk copies in the next
        asm volatile("fence.proxy.async;" ::: "memory");
        __syncthreads();
        if (abort_sh) {
            ok = false;
            mono_fail(a.bar);
            break;
        }
        // phase B reads own points only: its first slabs are fetched while alpha is reduced
        const int slabs = nload - 2;
        if (tid == kProducer) {
            fence_proxy_async_global();
            if (pend == nullptr)
                for (int e = 0; e < kDepth2 && e < slabs; e++) update_issue<2>(a, q2, own, e, nullptr, nullptr, nullptr);
            else
                for (int e = 0; e < kDepth5 && e < slabs; e++) update_issue<5>(a, q5, own, e, X, pend, pnew);
        }
        stamp_it(a, iter, 0);
        ok = reduce<1, 0>(pap, m0, a, epoch, seq);
        stamp_it(a, iter, 1);
        if (!ok) break;
        const double alpha = rv / pap[0];

        // phase B: r += alpha Ap, <r, r>, max |r|; in every second iteration x too, for the
        // direction before (which phase A has only read) and this one
        double sums[2] = {0.0, 0.0}, rmax[1] = {0.0};
        if (pend == nullptr) {
            update_own<KIND, 2>(a, q2, own, nullptr, nullptr, 0.0, nullptr, alpha, sums, rmax, &abort_sh);
            pend = pnew;
            apend = alpha;
        } else {
            update_own<KIND, 5>(a, q5, own, X, pend, apend, pnew, alpha, sums, rmax, &abort_sh);
            pend = nullptr;
        }
        asm volatile("fence.proxy.async;" ::: "memory");  // r is read by TMA next
        __syncthreads();
        if (abort_sh) {
            ok = false;
            mono_fail(a.bar);
            break;
        }
        stamp_it(a, iter, 2);
        ok = reduce<2, 1>(sums, rmax, a, epoch, seq);
        stamp_it(a, iter, 3);
        if (!ok) break;
        if (rmax[0] <= a.tol) {
            result = (int)iter;
            break;
        }
        const double rnv = KIND == PC_IMPLICIT ? -sums[0] / 6.0 : sums[1];
        beta = rnv / rv;
        rv = rnv;
        iter++;
        pold = pnew;
        pnew = (pnew == a.p0) ? a.p1 : a.p0;
    }

    if (ok && pend != nullptr) {
        for_own(a, own, [&](int i, int j, int k) {
            const long c = ((long)i * n + j) * n + k;
            X[c] = X[c] + apend * pend[c];
        });
    }
    __syncthreads();  // the pass below reads what other threads of the CTA wrote
    if (ok && a.prog == PROG_MAZE_LCG) {  // phi -= y (verlet.c:65)
        for_own(a, own, [&](int i, int j, int k) {
            const long c = ((long)i * n + j) * n + k;
            a.phi_new[c] = a.phi_new[c] + -1.0 * a.y[c];
        });
    }
    if (!ok && tid == kProducer) {
        // copies that may still be in flight into this CTA's shared memory: of each ring only
        // the last ones issued can be (bounded waits)
        for (int sq = max(0, ld - S); sq < ld; sq++) mbar_wait(&full[sq % S], (uint32_t)((sq / S) & 1));
        for (int sq = max(0, q2.issued - kDepth2); sq < q2.issued; sq++)
            mbar_wait(&q2.full[sq % kDepth2], (uint32_t)((sq / kDepth2) & 1));
        for (int sq = max(0, q5.issued - kDepth5); sq < q5.issued; sq++)
            mbar_wait(&q5.full[sq % kDepth5], (uint32_t)((sq / kDepth5) & 1));
    }
    __syncthreads();
    if (blockIdx.x == 0 && tid == 0) {
        a.result[0] = result;
        a.result[1] = ok ? 0 : 1;
    }
}

PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

}  // namespace

bool encode_grid_map(CUtensorMap* map, const double* base, int n, int bx, int by) {
    if (!g_encode) {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || fn == nullptr)
            return false;
        g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    const cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)n};
    const cuuint64_t strides[2] = {(cuuint64_t)n * 8, (cuuint64_t)n * n * 8};
    const cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(base), dims,
                                strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

bool cg_fast_supported(int n) { return n % 16 == 0 && n >= 16 && n <= 256; }

namespace {

// The cut of the grid into nj x ni blocks, at most one per SM: the CTAs march through the
// planes in step, so the halo rows that a block reads of its neighbours are in L2 then.
// (With 8-row blocks dealt out as one run of items the neighbours were half a sweep apart,
// and the halo, 2/8 of p and r, came from memory again.) At least two blocks along j, at most
// one column pair per thread; the cost counts the nine grid passes of an iteration and, at a
// tenth, the halo.
struct Plan {
    int rows, nj, ni, stages;
    size_t smem;
};
size_t plan_smem(int n, int rows, int stages) {
    const size_t slab = (size_t)(rows + 2) * n, a = (2 * stages + 2) * slab, b = (size_t)10 * rows * n;
    return (std::max(a, b) + (size_t)stages * 2 * n) * sizeof(double) + stages * sizeof(uint64_t) + 128;
}
Plan cg_fast_plan(int n, int sms) {
    constexpr size_t kBudget = 222 * 1024;  // of the 227 KB a CTA may use, beside its static 3.3 KB
    Plan best{};
    double cost = 1e300;
    for (int nj = 2; nj <= n && nj <= sms; nj++) {
        const int rows = (n + nj - 1) / nj, ni = std::min(sms / nj, n), planes = (n + ni - 1) / ni;
        if (rows * n > 2 * kProducer || plan_smem(n, rows, 3) > kBudget) continue;
        const double c = 9.0 * rows * planes + (rows + 2) * (planes + 2) - rows * planes + 18.0 * planes;
        if (c >= cost) continue;
        cost = c;
        best = Plan{rows, nj, ni, 3, 0};
    }
    if (best.rows == 0) return best;
    while (best.stages < kMaxStages && plan_smem(n, best.rows, best.stages + 1) <= kBudget) best.stages++;
    best.smem = plan_smem(n, best.rows, best.stages);
    return best;
}

int g_fast_device = -1;
int g_fast_blocks = 0;
}  // namespace

// Launch a CG program on the TMA path. Returns false if the path is unavailable here
// (caller falls back to the general engine).
bool cg_fast_launch(const EngineArgs& e, cudaStream_t stream) {
    static const bool verbose = getenv("MZB_PHASE_TIMING") != nullptr;
    auto no = [&](const char* why) {
        if (verbose) fprintf(stderr, "[cg fast path unavailable: %s]\n", why);
        return false;
    };
    const int n = e.n;
    if (e.pb) return no("Poisson-Boltzmann operator");
    if (!cg_fast_supported(n)) return no("grid size");
    const bool cg_prog = e.prog == PROG_CG || e.prog == PROG_PCG || e.prog == PROG_INIT_FIELD ||
                         e.prog == PROG_LCG_UPDATE || e.prog == PROG_MAZE_LCG;
    if (!cg_prog) return false;
    if ((e.prog == PROG_PCG || e.prog == PROG_MAZE_LCG) && e.precond != PC_IMPLICIT && e.precond != PC_JACOBI)
        return false;
    int dev;
    MZB_CHECK(cudaGetDevice(&dev));
    if (g_fast_device != dev) {
        int smem_max = 0;
        MZB_CHECK(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        smem_max -= 4096;  // static shared memory
        const void* kernels[2] = {(const void*)cg_fast_kernel<PC_IMPLICIT>, (const void*)cg_fast_kernel<PC_JACOBI>};
        int sms = 0;
        MZB_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        for (const void* kf : kernels) {
            MZB_CHECK(cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
            int per_sm = 0;
            MZB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kf, kThreads, smem_max));
            if (per_sm < 1) {
                if (verbose) {
                    cudaFuncAttributes fa;
                    cudaFuncGetAttributes(&fa, kf);
                    fprintf(stderr, "[cg fast: regs %d static smem %zu max threads %d, dyn smem %d]\n", fa.numRegs,
                            fa.sharedSizeBytes, fa.maxThreadsPerBlock, smem_max);
                }
                return no("occupancy 0");
            }
        }
        g_fast_device = dev;
        g_fast_blocks = sms;
    }
    // 16-byte accesses, and bulk copies that start on 16-byte boundaries
    for (const void* q : {(const void*)e.phi_new, (const void*)e.y, (const void*)e.x, (const void*)e.r, (const void*)e.p0,
                          (const void*)e.p1, (const void*)e.Ap})
        if ((uintptr_t)q & 15) return no("alignment");
    const Plan plan = cg_fast_plan(n, g_fast_blocks);
    if (plan.rows == 0) return no("no cut of the grid fits");
    CgFastArgs a{};
    a.prog = e.prog == PROG_PCG ? PROG_CG : e.prog;
    a.kind = (e.prog == PROG_PCG || e.prog == PROG_MAZE_LCG) ? e.precond : PC_IMPLICIT;
    a.n = n;
    a.rows = plan.rows;
    a.nj = plan.nj;
    a.ni = plan.ni;
    a.stages = plan.stages;
    a.tol = e.tol;
    a.c = e.c;
    a.q = e.q; a.phi_old = e.phi_old; a.phi_prev = e.phi_prev; a.phi_new = e.phi_new; a.y = e.y;
    a.b = e.b; a.x0 = e.x0; a.x = e.x;
    a.r = e.r; a.p0 = e.p0; a.p1 = e.p1; a.Ap = e.Ap; a.tmp = e.tmp;
    a.partials = e.partials; a.bar = e.bar; a.result = e.result;
    a.stamps = e.stamps;
    CUtensorMap mr, mrs, mp0, mp0s, mp1, mp1s;
    if (!encode_grid_map(&mr, a.r, n, n, 1) || !encode_grid_map(&mp0, a.p0, n, n, 1) ||
        !encode_grid_map(&mp1, a.p1, n, n, 1) || !encode_grid_map(&mrs, a.r, n, n, plan.rows + 2) ||
        !encode_grid_map(&mp0s, a.p0, n, n, plan.rows + 2) || !encode_grid_map(&mp1s, a.p1, n, n, plan.rows + 2))
        return no("tensor map encode");
    MZB_CHECK(cudaMemsetAsync(a.bar, 0, sizeof(GridBarrier), stream));
    void* params[] = {&mr, &mrs, &mp0, &mp0s, &mp1, &mp1s, &a};
    count_launch();
    const void* kf = a.kind == PC_JACOBI ? (const void*)cg_fast_kernel<PC_JACOBI> : (const void*)cg_fast_kernel<PC_IMPLICIT>;
    MZB_CHECK(cudaLaunchCooperativeKernel(kf, dim3(plan.nj * plan.ni), dim3(kThreads), params, plan.smem, stream));
    return true;
}

}  // namespace mzb
