// Conjugate-gradient field solves whose vectors stay on the SMs (sm_100a), for even grids of
// 16 to 128 points per side: small enough that every CTA holds its share of the direction p,
// halo included, in shared memory and its share of r, x and A p in tensor memory.
//
// Why. At these sizes a CG iteration moves little data, and what the streaming kernels
// (cg_fast.cu, engine.cu) spent was latency: two grid reductions of 2.2 us each (arrive,
// poll, then one more trip to gather the partial sums) and two passes that fetch every
// vector through L2 again. Here:
//   - the grid's rows (i, j) are cut into Pi x Pj patches of whole rows, one CTA each, so the
//     k neighbours (and their periodic wrap) stay inside a row and the halo is whole rows;
//   - p sits in shared memory with its halo rows. r, x and A p sit in tensor memory, 256 KB
//     per SM that no other work of this library uses, read and written by the thread that
//     owns the points (tcgen05.ld / tcgen05.st): with p they are more than registers and
//     shared memory can hold above 100^3, and held in registers they forced every loop over
//     a thread's points to be unrolled and spilled. Above 10 pairs per thread x stays in the
//     grid array;
//   - only the patch's edge rows of r travel. Each value goes out as 16 bytes {value, step}
//     in one store; the reader polls the value itself until the step matches, so the
//     exchange needs no fence, no flag and no second trip. Two buffers alternate: a CTA can
//     write step s + 2 only after its neighbours sent s + 1, which they do after reading s;
//   - the two scalar products of an iteration are summed in fixed point (fast_sum): one
//     relaxed add per CTA into two words that carry the arrival count beside the value, so
//     the poll that sees the last arrival already has the sum, whatever the order of
//     arrival (0.93 us against 2.2 us on 148 CTAs).
// The arithmetic per point is the reference's (operation order, every product rounded); only
// the sums over points are taken in another, fixed, order.
//
// Measured on one B200, us per iteration, before (cg_fast.cu at 16 n, else engine.cu) and now:
// Laplacian 16^3 12.7 / 4.7, 64^3 14.5 / 5.0, 80^3 20.4 / 6.4, 100^3 29.6 / 9.2, 128^3 38.4 /
// 15.6; Poisson-Boltzmann 64^3 14.2 / 5.9, 96^3 31.0 / 11.3, 128^3 53.4 / 20.9. Bound by
// latency: at 64^3 two sums and a halo trip take 2.6 us, the rest is short dependent chains of
// 4 warps per scheduler; at 128^3 issue and the shared-memory reads of the stencil (3.6 us) and
// the L2 round trips of x (2.6 us). Register spills are what it cannot afford, since with the
// shared memory taken they land in L2: batches of 4 pairs instead of 2, or 4 instead of 2 halo
// pairs in flight, spilled 100 to 600 bytes and cost 20 to 160 %.
#include <algorithm>
#include <atomic>

#include "resident.cuh"

namespace mzb {
namespace {

typedef unsigned long long u64;

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kMaxHaloSteps = 4;   // halo rows one warp receives at most
constexpr int kTmemColumns = 512;  // all of tensor memory; each warp owns 128 columns of its 32 lanes
constexpr int kBatch = 2;          // pairs whose vectors a thread has in flight together
constexpr int kApply = 2;          // pairs of the Laplacian worked together (3 and 4: within 6 % slower)

// Head of the work area, zeroed before every launch; the halo buffers follow it.
struct alignas(128) RedWords {
    u64 lo, hi;
};
struct ResHeader {
    alignas(128) GridBarrier bar;
    RedWords red[2];
};

struct ResArgs {
    EngineArgs e;
    int Pi, Pj, cap;   // patches along i and j; elements of one halo strip
    int pairs;         // the most pairs any thread has
    int cPi, cPj, cpairs, coarse_at;  // the coarse grid's patches and its plane in shared memory (multigrid)
    int smem_doubles;  // dynamic shared memory
    int x_tmem;        // x in tensor memory (else in the grid array it ends in)
    u64 step0;         // halo step numbers of this launch start above this
    ResHeader* head;
    ulonglong2* strips;  // [CTA][2][4][cap] {value bits, step}
};

__device__ __forceinline__ void st_pair(ulonglong2* p, double v, u64 step) {
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(step)
                 : "memory");
}
__device__ __forceinline__ void ld_pair(const ulonglong2* p, u64& a, u64& b) {
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void red_add(u64* p, u64 v) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The CTA's shared memory: its state, the plane of p, the received halo rows of r.
struct Shared {
    double sum[kWarps];  // block reductions
    double res[2];       // a grid-wide sum and its mark count or maximum
    u64 lo[2], hi[2];    // the fixed-point words' values after their last use
    int flag[2];         // [0] a wait ran out, [1] outcome of the last fast_sum
    int nb[2][4];        // CTAs of the patches at i - 1, i + 1, j - 1, j + 1; [1]: the coarse grid's
    uint32_t tmem;
    unsigned bulk[kWarps];  // multigrid: bulk_units of the fine grid
};
constexpr int kStateDoubles = 48;
static_assert(sizeof(Shared) <= kStateDoubles * sizeof(double), "state area");
extern __shared__ __align__(128) double smem[];
__device__ __forceinline__ Shared& shared_state() { return *reinterpret_cast<Shared*>(smem); }

// One CTA's patch of rows, i in [i0, i0 + bi), j in [j0, j0 + bj), whole rows of n points,
// worked as pairs (k, k + 1). A thread owns one column of pairs (lj, kk) and `cnt` consecutive
// li of it, from li0 on: the i neighbours of its pairs are its own, the k neighbours lie in
// the lanes beside it, and unit m's place in a plane or a grid is the first one's plus m
// pitches. S threads share a column, each at most SL pairs long. Shared planes hold
// (bi + 2) x (bj + 2) rows, row (li + 1) (bj + 2) + lj + 1.
struct Patch {
    int n, h, i0, bi, j0, bj, pitch;  // pitch: doubles from row li to li + 1 of a plane
    int li0, cnt, lj, kk;             // this thread's pairs (cnt = 0: none)
    int o0;                           // its first pair's place in a plane
    int g0, n2;                       // and in the grid; n^2
    int coarse;                       // 1: a patch of the coarse grid (Shared::nb)
};
__device__ __forceinline__ Patch make_patch(int n, int Pi, int Pj, int coarse) {
    Patch p;
    p.coarse = coarse;
    p.n = n;
    p.h = n / 2;
    p.n2 = n * n;
    const int a = blockIdx.x / Pj, b = blockIdx.x - a * Pj;
    if (a >= Pi) {  // a CTA without a patch (coarse grids): no points, no neighbours
        p.i0 = p.j0 = p.bi = p.bj = 0;
        p.pitch = 2 * n;
        p.li0 = p.cnt = p.lj = p.kk = 0;
        p.o0 = 0;
        p.g0 = 0;
        return p;
    }
    p.i0 = a * n / Pi;
    p.bi = (a + 1) * n / Pi - p.i0;
    p.j0 = b * n / Pj;
    p.bj = (b + 1) * n / Pj - p.j0;
    p.pitch = (p.bj + 2) * n;
    if (threadIdx.x == 0) {
        int* nb = shared_state().nb[coarse];
        nb[0] = (a == 0 ? Pi - 1 : a - 1) * Pj + b;
        nb[1] = (a + 1 == Pi ? 0 : a + 1) * Pj + b;
        nb[2] = a * Pj + (b == 0 ? Pj - 1 : b - 1);
        nb[3] = a * Pj + (b + 1 == Pj ? 0 : b + 1);
    }
    const int C = p.bj * p.h, S = kThreads / C, SL = (p.bi + S - 1) / S;
    const int seg = threadIdx.x / C, col = threadIdx.x - seg * C;
    p.lj = col / p.h;
    p.kk = col - p.lj * p.h;
    p.li0 = seg * SL;
    p.cnt = p.bi - p.li0;
    if (seg >= S || p.cnt < 0) p.cnt = 0;
    if (p.cnt > SL) p.cnt = SL;
    if (p.cnt == 0) p.li0 = 0;  // reads in bounds
    p.o0 = ((p.li0 + 1) * (p.bj + 2) + p.lj + 1) * n + 2 * p.kk;
    p.g0 = ((p.i0 + p.li0) * n + p.j0 + p.lj) * n + 2 * p.kk;
    return p;
}
// Rows of a plane along i: the patch's, its two halo rows and room for the slots past the last
// units (read for nothing, never written).
__host__ __device__ __forceinline__ int plane_rows(int n, int bi, int bj, int units) {
    const int S = bj > 0 ? kThreads / (bj * (n / 2)) : 1, SL = (bi + S - 1) / S;
    return (S - 1) * SL + units + 2;
}

__device__ __forceinline__ double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st2(double* p, double2 v) { *reinterpret_cast<double2*>(p) = v; }

// ------------------------------------------------------------------------------------
// Tensor memory as the threads' own storage: a warp reaches 32 lanes (one per thread) and
// here 128 columns of 32 bits, i.e. 32 pairs of doubles per thread. Every access is made by
// the whole warp.
// ------------------------------------------------------------------------------------
struct Cell {
    uint32_t a, b, c, d;
};
__device__ __forceinline__ void tm_load(Cell& v, uint32_t at) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.a), "=r"(v.b), "=r"(v.c), "=r"(v.d)
                 : "r"(at));
}
// The loads' results may be used after this; the operands tie them to it.
template <int N>
__device__ __forceinline__ void tm_loaded(Cell (&v)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < N; q++) asm volatile("" : "+r"(v[q].a), "+r"(v[q].b), "+r"(v[q].c), "+r"(v[q].d));
}
__device__ __forceinline__ void tm_store(uint32_t at, double2 v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(__double2loint(v.x)),
                 "r"(__double2hiint(v.x)), "r"(__double2loint(v.y)), "r"(__double2hiint(v.y)));
}
__device__ __forceinline__ void tm_stored() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ double2 pair_of(const Cell& v) {
    return make_double2(__hiloint2double((int)v.b, (int)v.a), __hiloint2double((int)v.d, (int)v.c));
}
// All of the SM's tensor memory (the CTA is alone on its SM); every exit path frees it.
__device__ __forceinline__ uint32_t tm_alloc(uint32_t* slot) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(slot)),
                     "n"(kTmemColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return *slot;
}
__device__ __forceinline__ void tm_free(uint32_t base) {
    tm_stored();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(kTmemColumns) : "memory");
}
// Column 0 of this warp's share.
__device__ __forceinline__ uint32_t tm_own(uint32_t base) {
    const uint32_t w = threadIdx.x >> 5;
    return base + ((w & 3u) << 21) + (w >> 2) * 128u;
}

// ------------------------------------------------------------------------------------
// Grid-wide sums.
// ------------------------------------------------------------------------------------
struct Ctl {
    int seq = 0;       // reductions through the fixed-point words
    int slow_seq = 0;  // reductions through the partials
    u64 step;          // halo step number last published
};

// Sum of v over the block in thread 0 (fixed tree); true in every thread if `any` held in one.
__device__ __forceinline__ bool block_total(double& v, bool any) {
    Shared& sh = shared_state();
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh.sum[threadIdx.x >> 5] = v;
    const bool r = __syncthreads_or(any);
    if (threadIdx.x < kWarps) {
        v = sh.sum[threadIdx.x];
#pragma unroll
        for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync((1u << kWarps) - 1u, v, o);
    }
    return r;
}

// Sum of s and maximum of m over the grid through per-CTA partials and a grid barrier: the
// way for values of any size (first use of a sum, one that grew or shrank too much for fast_sum).
struct Reduced {
    double sum, max;
    bool ok;
};
__device__ __noinline__ Reduced slow_reduce(const ResArgs& a, int slow_seq, double s, double m) {
    Shared& sh = shared_state();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int G = gridDim.x;
    double v = warp_sum(s), x = warp_max(m);
    __syncthreads();
    if (lane == 0) sh.sum[w] = v;
    __syncthreads();
    if (w == 0) v = warp_sum(lane < kWarps ? sh.sum[lane] : 0.0);
    __syncthreads();
    if (lane == 0) sh.sum[w] = x;
    __syncthreads();
    if (w == 0) x = warp_max(lane < kWarps ? sh.sum[lane] : 0.0);
    double* part = a.e.partials + (slow_seq & 1) * 2 * G;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = v;
        part[G + blockIdx.x] = x;
    }
    const bool ok = grid_sync(&a.head->bar);
    if (w == 0) {
        v = 0.0;
        x = 0.0;
        for (int b = lane; b < G; b += 32) {
            v += __ldcg(part + b);
            x = fmax(x, __ldcg(part + G + b));
        }
        v = warp_sum(v);
        x = warp_max(x);
        if (lane == 0) {
            sh.res[0] = v;
            sh.res[1] = x;
        }
    }
    __syncthreads();
    const Reduced r = {sh.res[0], sh.res[1], ok};
    __syncthreads();
    return r;
}

// Thread 0's part of a grid-wide sum in fixed point: post, then wait. The CTA's value, scaled by a power of
// two that puts the sum's previous value `prev` at 2^22, is added as an integer part
// (32 bits, offset) to `hi` and a fraction (48 bits) to `lo`; bits 56.. of both words count
// the arrivals, bits 40.. of `hi` the CTAs that raised `mark` and bits 48.. those whose value
// does not fit (more than 512 times the previous sum, or not finite). Integer addition does
// not depend on the order, the words are never cleared (each use subtracts the value after
// the one before; two words alternate, so a word is read by all before it is used again).
// Up to 148 fractions rounded to 2^-48 leave an error below 2^-41.7 in a sum whose predecessor
// stands at 2^22: less than FP64 rounds away itself unless the sum has shrunk by more than 2^11
// (a smooth right-hand side can take it to 2^-100 in one iteration), and then it is taken
// through the partials. The wait returns 0: the sum is in res[0] and the marks in res[1]; 1: a
// value did not fit or the sum is too small (all CTAs read the same words); -1: it ran out of
// time.
constexpr long long kSmallestSum = 1 << 11;
struct Posted {
    double inv_scale;
};
__device__ __forceinline__ Posted fast_sum_post(const ResArgs& a, int seq, double v, double prev, bool mark) {
    RedWords* w = &a.head->red[seq & 1];
    const long long ex = (__double_as_longlong(prev) >> 52) & 0x7ff;  // 1023 + exponent
    const double t = v * __longlong_as_double((2 * 1023 + 22 - ex) << 52);
    u64 hi = (u64)1 << 56, lo = (u64)1 << 56;
    if (fabs(t) < 2147483000.0) {
        const double f = floor(t);
        hi += (u64)((long long)f + (1ll << 31));
        lo += __double2ull_rn((t - f) * 0x1p48);
    } else {
        hi += (u64)1 << 48;
    }
    if (mark) hi += (u64)1 << 40;
    red_add(&w->lo, lo);
    red_add(&w->hi, hi);
    return {__longlong_as_double((ex - 22) << 52)};
}
__device__ __forceinline__ int fast_sum_wait(const ResArgs& a, int seq, const Posted& posted) {
    Shared& sh = shared_state();
    const int s = seq & 1;
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(&a.head->red[s]);
    const u64 G = gridDim.x, lo0 = sh.lo[s], hi0 = sh.hi[s];
    u64 x, y, dl, dh;
    unsigned polls = 0;
    u64 t0 = 0;
    for (;;) {
        ld_pair(w, x, y);
        dl = x - lo0;
        dh = y - hi0;
        if ((dl >> 56) == G && (dh >> 56) == G) break;
        if ((++polls & 255u) == 0u) {
            const u64 now = global_ns();
            if (t0 == 0) t0 = now;
            if (ld_acquire_u32(&a.head->bar.err) != 0u || now - t0 > kBarrierTimeoutNs) {
                atomicOr(&a.head->bar.err, 1u);
                return -1;
            }
        }
    }
    sh.lo[s] = x;
    sh.hi[s] = y;
    const long long whole = (long long)(dh & (((u64)1 << 40) - 1)) - (long long)(G << 31);
    const double F = (double)(dl & (((u64)1 << 56) - 1)) * 0x1p-48;
    sh.res[0] = ((double)whole + F) * posted.inv_scale;
    sh.res[1] = (double)((dh >> 40) & 0xff);
    // the fractions add less than G + 1 to the whole part; no branch, all warps wait for this
    const bool small = (u64)(whole + kSmallestSum + (long long)G) < (u64)(2 * kSmallestSum + (long long)G);
    return (int)(small | (((dh >> 48) & 0xff) != 0));
}
__device__ __forceinline__ bool fixed_point_ok(double prev) {
    const int ex = (int)((__double_as_longlong(prev) >> 52) & 0x7ff);
    return ex > 64 && ex < 2000;
}

// ------------------------------------------------------------------------------------
// Halo exchange of one value per point of the patch's edge rows.
// ------------------------------------------------------------------------------------
// First element of a CTA's strip `side` for a step (the buffers hold fewer than 2^31 elements).
__device__ __forceinline__ int strip(const ResArgs& a, int cta, u64 step, int side) {
    return ((cta * 2 + (int)(step & 1)) * 4 + side) * a.cap;
}
// Publish unit m's pair if it lies in an edge row: strips 0, 1 hold rows li = 0 and bi - 1
// (by lj), 2, 3 hold lj = 0 and bj - 1 (by li).
__device__ __forceinline__ void publish(const ResArgs& a, const Patch& p, int m, double2 v, u64 step) {
    const int li = p.li0 + m, k = 2 * p.kk;
    const bool e0 = li == 0, e1 = li == p.bi - 1, e2 = p.lj == 0, e3 = p.lj == p.bj - 1;
    if (!(e0 | e1 | e2 | e3)) return;
    ulonglong2* mine = a.strips + strip(a, blockIdx.x, step, 0) + k;
    auto put = [&](int side, int row) {
        ulonglong2* d = mine + side * a.cap + row * p.n;
        st_pair(d, v.x, step);
        st_pair(d + 1, v.y, step);
    };
    if (e0) put(0, p.lj);
    if (e1) put(1, p.lj);
    if (e2) put(2, li);
    if (e3) put(3, li);
}
// Halo row x of the patch (0 .. 2 bi + 2 bj): where it comes from and its place in a shared
// plane. Rows: li = -1, li = bi (by lj), lj = -1, lj = bj (by li).
__device__ __forceinline__ int halo_rows(const Patch& p) { return 2 * (p.bi + p.bj); }
__device__ __forceinline__ int halo_source(const ResArgs& a, const Patch& p, int x, u64 step) {
    const bool along_j = x < 2 * p.bj;
    const int len = along_j ? p.bj : p.bi, y = along_j ? x : x - 2 * p.bj;
    const bool hi = y >= len;
    const int cta = shared_state().nb[p.coarse][(along_j ? 0 : 2) + (hi ? 1 : 0)];
    const int side = (along_j ? 0 : 2) + (hi ? 0 : 1);
    return strip(a, cta, step, side) + (hi ? y - len : y) * p.n;
}
__device__ __forceinline__ int halo_at(const Patch& p, int x) {
    const bool along_j = x < 2 * p.bj;
    const int len = along_j ? p.bj : p.bi, y = along_j ? x : x - 2 * p.bj;
    const bool hi = y >= len;
    const int at = hi ? y - len : y, far = hi ? (along_j ? p.bi : p.bj) : -1;
    const int li = along_j ? far : at, lj = along_j ? at : far;
    return ((li + 1) * (p.bj + 2) + lj + 1) * p.n;
}
// Receive a thread's pairs of a halo row (null: none); false when the wait ran out.
template <int NB>
__device__ __forceinline__ bool receive(const ResArgs& a, const ulonglong2* const (&src)[NB], u64 step, double2 (&v)[NB]) {
    unsigned polls = 0;
    u64 t0 = 0;
    for (;;) {
        u64 x[NB], xs[NB], y[NB], ys[NB];
#pragma unroll
        for (int q = 0; q < NB; q++) {
            xs[q] = ys[q] = step;
            x[q] = y[q] = 0;
            if (src[q] != nullptr) {
                ld_pair(src[q], x[q], xs[q]);
                ld_pair(src[q] + 1, y[q], ys[q]);
            }
        }
        bool all = true;
#pragma unroll
        for (int q = 0; q < NB; q++) {
            all = all && xs[q] == step && ys[q] == step;
            v[q] = make_double2(__longlong_as_double(x[q]), __longlong_as_double(y[q]));
        }
        if (all) return true;
        if ((++polls & 255u) == 0u) {
            const u64 now = global_ns();
            if (t0 == 0) t0 = now;
            if (ld_acquire_u32(&a.head->bar.err) != 0u || now - t0 > kBarrierTimeoutNs) {
                atomicOr(&a.head->bar.err, 1u);
                return false;
            }
        }
    }
}

// k parity of colour's points in halo row x.
__device__ __forceinline__ int halo_parity(const Patch& p, int x, int colour) {
    const bool along_j = x < 2 * p.bj;
    const int len = along_j ? p.bj : p.bi, y = along_j ? x : x - 2 * p.bj;
    const bool hi = y >= len;
    const int at = hi ? y - len : y, far = hi ? (along_j ? p.bi : p.bj) : -1;
    return (p.i0 + p.j0 + at + far + colour) & 1;
}
// Wait for NB single values of step `step` at strips + src[q] (negative: none).
template <int NB>
__device__ __forceinline__ bool receive_values(const ResArgs& a, const int (&src)[NB], u64 step, u64 (&x)[NB]) {
    unsigned polls = 0;
    u64 t0 = 0;
    for (;;) {
        u64 xs[NB];
#pragma unroll
        for (int q = 0; q < NB; q++) {
            xs[q] = step;
            if (src[q] >= 0) ld_pair(a.strips + src[q], x[q], xs[q]);
        }
        bool all = true;
#pragma unroll
        for (int q = 0; q < NB; q++) all = all && xs[q] == step;
        if (all) return true;
        if ((++polls & 255u) == 0u) {
            const u64 now = global_ns();
            if (t0 == 0) t0 = now;
            if (ld_acquire_u32(&a.head->bar.err) != 0u || now - t0 > kBarrierTimeoutNs) {
                atomicOr(&a.head->bar.err, 1u);
                return false;
            }
        }
    }
}

// ------------------------------------------------------------------------------------
// Operators on a shared plane: a pair of A p at plane offset o from the pairs im, c, ip at
// li - 1, li, li + 1 (carried along the column). The k neighbours come from the lanes beside,
// at a row's ends and the warp's edges from the plane.
// ------------------------------------------------------------------------------------
struct Coef {
    const double *ex, *ey, *ez, *dg;
    double eb, db;  // face coefficient and diagonal of the grid's corner, taken for the bulk's
};
// The Poisson-Boltzmann coefficients around one pair.
struct Faces {
    double2 exc, exm, eyc, eym, ezc, dg;
    double ezm;
};
__device__ __forceinline__ Faces bulk_faces(const Coef& cf) {
    Faces f;
    f.exc = f.exm = f.eyc = f.eym = f.ezc = make_double2(cf.eb, cf.eb);
    f.dg = make_double2(cf.db, cf.db);
    f.ezm = cf.eb;
    return f;
}
__device__ __forceinline__ Faces load_faces(const Patch& p, const Coef& cf, int m) {
    const int q = m < p.cnt ? m : p.cnt > 0 ? p.cnt - 1 : 0, n = p.n;
    const int g = p.g0 + q * p.n2;
    Faces f;
    f.exc = ld2(cf.ex + g);
    f.eyc = ld2(cf.ey + g);
    f.ezc = ld2(cf.ez + g);
    f.dg = ld2(cf.dg + g);
    f.exm = ld2(cf.ex + g + (p.i0 + p.li0 + q == 0 ? (n - 1) * p.n2 : -p.n2));
    f.eym = ld2(cf.ey + g + (p.j0 + p.lj == 0 ? (n - 1) * n : -n));
    f.ezm = cf.ez[g + (p.kk == 0 ? n - 1 : -1)];
    return f;
}
struct Around {
    double km, kp;
    double2 jp, jm;
};
__device__ __forceinline__ Around around(const Patch& p, const double* P, int o, double2 c) {
    const int n = p.n, lane = threadIdx.x & 31;
    const bool start = p.kk == 0, end = p.kk == p.h - 1;
    Around t;
    t.km = __shfl_up_sync(0xffffffffu, c.y, 1);
    t.kp = __shfl_down_sync(0xffffffffu, c.x, 1);
    if (start || lane == 0) t.km = P[start ? o + n - 1 : o - 1];
    if (end || lane == 31) t.kp = P[end ? o + 2 - n : o + 2];
    t.jp = ld2(P + o + n);
    t.jm = ld2(P + o - n);
    return t;
}
__device__ __forceinline__ double2 apply_lap(const Around& t, double2 im, double2 c, double2 ip) {
    double s0 = ip.x + im.x;
    s0 = s0 + t.jp.x;
    s0 = s0 + t.jm.x;
    s0 = s0 + c.y;
    s0 = s0 + t.km;
    double s1 = ip.y + im.y;
    s1 = s1 + t.jp.y;
    s1 = s1 + t.jm.y;
    s1 = s1 + t.kp;
    s1 = s1 + c.x;
    return make_double2(s0 - c.x * 6.0, s1 - c.y * 6.0);
}
__device__ __forceinline__ double2 apply_pb(const Around& t, double2 im, double2 c, double2 ip, const Faces& f) {
    double s0 = ip.x * f.exc.x + im.x * f.exm.x;
    s0 = s0 + t.jp.x * f.eyc.x;
    s0 = s0 + t.jm.x * f.eym.x;
    s0 = s0 + c.y * f.ezc.x;
    s0 = s0 + t.km * f.ezm;
    double s1 = ip.y * f.exc.y + im.y * f.exm.y;
    s1 = s1 + t.jp.y * f.eyc.y;
    s1 = s1 + t.jm.y * f.eym.y;
    s1 = s1 + t.kp * f.ezc.y;
    s1 = s1 + c.x * f.ezc.x;
    return make_double2(s0 - c.x * f.dg.x, s1 - c.y * f.dg.y);
}
// Bit m: every coefficient around unit m of every lane of this warp equals the bulk's, so the
// constants stand for the loads (most of the solvent away from the ions; found once per solve).
__device__ __forceinline__ unsigned bulk_units(const Patch& p, const Coef& cf, int units) {
    unsigned mask = 0;
    for (int m = 0; m < units; m++) {
        bool same = true;
        if (m < p.cnt) {
            const Faces f = load_faces(p, cf, m);
            const double2 v[5] = {f.exc, f.exm, f.eyc, f.eym, f.ezc};
#pragma unroll
            for (int q = 0; q < 5; q++) same = same && v[q].x == cf.eb && v[q].y == cf.eb;
            same = same && f.dg.x == cf.db && f.dg.y == cf.db && f.ezm == cf.eb;
        }
        if (__all_sync(0xffffffffu, same)) mask |= 1u << m;
    }
    return mask;
}

// The same operator on a grid in global memory, value by value (set-up passes).
struct Nb {
    long c, ip, im, jp, jm, kp, km;
};
__device__ __forceinline__ Nb nb_of(int n, int i, int j, int k) {
    const long n2 = (long)n * n;
    Nb o;
    o.c = ((long)i * n + j) * n + k;
    o.ip = o.c + (i + 1 == n ? -(long)(n - 1) * n2 : n2);
    o.im = o.c + (i == 0 ? (long)(n - 1) * n2 : -n2);
    o.jp = o.c + (j + 1 == n ? -(long)(n - 1) * n : (long)n);
    o.jm = o.c + (j == 0 ? (long)(n - 1) * n : -(long)n);
    o.kp = o.c + (k + 1 == n ? -(long)(n - 1) : 1L);
    o.km = o.c + (k == 0 ? (long)(n - 1) : -1L);
    return o;
}
template <bool PB, class F>
__device__ __forceinline__ double apply_at(const Nb& o, const Coef& cf, F&& f) {
    if (!PB) {
        double s = f(o.ip) + f(o.im);
        s = s + f(o.jp);
        s = s + f(o.jm);
        s = s + f(o.kp);
        s = s + f(o.km);
        return s - f(o.c) * 6.0;
    }
    double s = f(o.ip) * cf.ex[o.c] + f(o.im) * cf.ex[o.im];
    s = s + f(o.jp) * cf.ey[o.c];
    s = s + f(o.jm) * cf.ey[o.jm];
    s = s + f(o.kp) * cf.ez[o.c];
    s = s + f(o.km) * cf.ez[o.km];
    return s - f(o.c) * cf.dg[o.c];
}

// The preconditioned residual as the direction's increment (see cg_fast.cu) and its term of
// <r, M^-1 r>. The Jacobi form's r / 6 is formed from the rounded reciprocal and one exact
// remainder (Markstein 1990), which rounds as the division does.
__device__ __forceinline__ double sixth(double r) {
    const double q = r * (1.0 / 6.0);
    return fma(fma(-6.0, q, r), 1.0 / 6.0, q);
}
template <int KIND>
__device__ __forceinline__ double zf(double r) {
    if (KIND == PC_IMPLICIT) return (1.0 / 6.0) * r;
    if (KIND == PC_JACOBI) return sixth(r);
    return -1.0 * r;
}
template <int KIND>
__device__ __forceinline__ double rz_term(double r) {
    if (KIND == PC_JACOBI) return r * -sixth(r);
    return r * r;
}

// Phase times (EngineArgs::stamps, a debug aid): slots 0 .. 2 the set-up, 4 + 4 it + {0 .. 3}
// the ends of p and A p, their sum, the update, its sum, of iteration it < kCgStampIters.
// Kernels of their own (TIMED): tested at run time in every phase they cost 3 % at 64^3.
template <bool TIMED>
__device__ __forceinline__ void stamp(const ResArgs& a, int slot) {
    if (TIMED && (blockIdx.x | threadIdx.x) == 0) a.e.stamps[slot] = global_ns();
}
template <bool TIMED>
__device__ __forceinline__ void stamp_it(const ResArgs& a, long iter, int k) {
    if (TIMED && iter < kCgStampIters) stamp<true>(a, 4 + 4 * (int)iter + k);
}

// ------------------------------------------------------------------------------------
// The iteration. On entry tensor memory holds the patch's residual (unit m at tr + 4 m) and
// x (tx + 4 m, or the grid at xg); rv is <r, z(r)> and r0 = max |r| (COARSE). Slots past a
// thread's last unit hold zeros. Returns the reference's value: conj_grad the 0-based
// iteration at convergence or -1, cg_coarse the number of iterations
// (library/src/plcg.c:28-238, multigrid.c:13-96, multigrid_pb.c:16-97).
// ------------------------------------------------------------------------------------
template <bool PB, int KIND, bool COARSE, int HL, bool TIMED>
__device__ __forceinline__ int iterate(const ResArgs& a, Ctl& c, const Patch& p, int units, double* P, uint32_t tr, uint32_t tap, uint32_t tx, double* xg,
                       const Coef& cf, double rv, double r0, double tol, long limit, bool& ok) {
    Shared& sh = shared_state();
    double* hs = P + plane_rows(p.n, p.bi, p.bj, units) * p.pitch;
    const double stop = COARSE ? tol * r0 : tol;
    // halo rows of r: warp v >= 1 takes rows v - 1, v + 14, ... and its lanes the row's pairs;
    // warp 0 waits for the sums
    const int wid = (int)(threadIdx.x >> 5) - 1, lane = threadIdx.x & 31, nh = halo_rows(p);
    const unsigned bulk = PB ? bulk_units(p, cf, units) : 0u;

    auto receive_halo = [&]() {
        if (wid < 0) return;
        constexpr int NR = HL == 1 ? 2 : 1;  // rows whose loads are out together
#pragma unroll 1
        for (int y = wid; y < nh; y += NR * (kWarps - 1)) {
            const ulonglong2* src[NR * HL];
            double2 v[NR * HL];
#pragma unroll
            for (int q = 0; q < NR; q++) {
                const int row = y + q * (kWarps - 1);
                const ulonglong2* at = a.strips + (row < nh ? halo_source(a, p, row, c.step) : 0) + 2 * lane;
#pragma unroll
                for (int t = 0; t < HL; t++)
                    src[q * HL + t] = row < nh && lane + 32 * t < p.h ? at + 64 * t : nullptr;
            }
            if (!receive<NR * HL>(a, src, c.step, v)) sh.flag[0] = 1;
#pragma unroll
            for (int q = 0; q < NR; q++)
#pragma unroll
                for (int t = 0; t < HL; t++)
                    if (src[q * HL + t] != nullptr)
                        st2(hs + (y + q * (kWarps - 1)) * p.n + 2 * (lane + 32 * t), v[q * HL + t]);
        }
    };

    c.step++;
#pragma unroll 1
    for (int m = 0; m < units; m++) {
        Cell r[1];
        tm_load(r[0], tr + 4 * m);
        tm_loaded(r);
        if (m < p.cnt) publish(a, p, m, pair_of(r[0]), c.step);
        __syncwarp();
    }
    receive_halo();

    long iter = 0;
    double beta = 0.0, pap_prev = 0.0, rr_prev = 0.0;
    while (iter < limit) {
        const bool first = iter == 0;
        // p <- beta p + z(r) on the patch and its halo
        auto direction = [&](double2 rr, double2 po) {
            double2 z = make_double2(zf<KIND>(rr.x), zf<KIND>(rr.y));
            if (!first) {
                z.x = po.x * beta + z.x;
                z.y = po.y * beta + z.y;
            }
            return z;
        };
#pragma unroll 1
        for (int m0 = 0; m0 < units; m0 += kBatch) {
            Cell r[kBatch];
            double2 po[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                tm_load(r[q], tr + 4 * min(m0 + q, units - 1));
                po[q] = ld2(P + p.o0 + min(m0 + q, units - 1) * p.pitch);
            }
            tm_loaded(r);
#pragma unroll
            for (int q = 0; q < kBatch; q++)
                if (m0 + q < p.cnt) st2(P + p.o0 + (m0 + q) * p.pitch, direction(pair_of(r[q]), po[q]));
            __syncwarp();
        }
        if (wid >= 0) {
#pragma unroll 1
            for (int y = wid; y < nh; y += kWarps - 1) {
                const int o = halo_at(p, y);
                double2 rr[HL], po[HL];
#pragma unroll
                for (int t = 0; t < HL; t++) {
                    const int k = min(2 * (lane + 32 * t), p.n - 2);
                    rr[t] = ld2(hs + y * p.n + k);
                    po[t] = ld2(P + o + k);
                }
#pragma unroll
                for (int t = 0; t < HL; t++) {
                    const int k = 2 * (lane + 32 * t);
                    if (k < p.n) st2(P + o + k, direction(rr[t], po[t]));
                }
                __syncwarp();
            }
        }
        __syncthreads();
        // A p, <p, A p>: kApply units of the column at a time, their loads before any sum
        double pap = 0.0;
        {
            double2 im = ld2(P + p.o0 - p.pitch), pc = ld2(P + p.o0);
            if (PB) {
                Faces next = (bulk & 1u) ? bulk_faces(cf) : load_faces(p, cf, 0);
#pragma unroll 1
                for (int m = 0; m < units; m++) {  // the next pair's coefficients are on their way meanwhile
                    const int o = p.o0 + m * p.pitch;
                    const Faces f = next;
                    if (m + 1 < units) next = ((bulk >> (m + 1)) & 1u) ? bulk_faces(cf) : load_faces(p, cf, m + 1);
                    const double2 ip = ld2(P + o + p.pitch);
                    const double2 v = apply_pb(around(p, P, o, pc), im, pc, ip, f);
                    __syncwarp();
                    tm_store(tap + 4 * m, v);
                    if (m < p.cnt) {
                        pap += pc.x * v.x;
                        pap += pc.y * v.y;
                    }
                    im = pc;
                    pc = ip;
                }
            } else {
#pragma unroll 1
                for (int m0 = 0; m0 < units; m0 += kApply) {
                    double2 col[kApply + 2];
                    Around t[kApply];
                    col[0] = im;
                    col[1] = pc;
#pragma unroll
                    for (int q = 0; q < kApply; q++) {
                        const int o = p.o0 + min(m0 + q, units - 1) * p.pitch;
                        col[q + 2] = ld2(P + o + p.pitch);
                        t[q] = around(p, P, o, col[q + 1]);
                    }
#pragma unroll
                    for (int q = 0; q < kApply; q++) {
                        const double2 v = apply_lap(t[q], col[q], col[q + 1], col[q + 2]);
                        __syncwarp();
                        if (m0 + q < units) tm_store(tap + 4 * (m0 + q), v);
                        if (m0 + q < p.cnt) {
                            pap += col[q + 1].x * v.x;
                            pap += col[q + 1].y * v.y;
                        }
                    }
                    im = col[kApply];
                    pc = col[kApply + 1];
                }
            }
        }
        stamp_it<TIMED>(a, iter, 0);
        int how = 1;
        if (fixed_point_ok(pap_prev)) {
            double v = pap;
            block_total(v, false);
            if (threadIdx.x == 0) {
                const Posted w = fast_sum_post(a, c.seq, v, pap_prev, false);
                sh.flag[1] = fast_sum_wait(a, c.seq, w);
            }
            __syncthreads();
            how = sh.flag[1];
            c.seq++;
            if (how == 0) pap = sh.res[0];
        }
        ok = how >= 0 && sh.flag[0] == 0;
        if (!ok) return -1;
        if (how == 1) {
            const Reduced d = slow_reduce(a, c.slow_seq++, pap, 0.0);
            pap = d.sum;
            ok = d.ok;
            if (!ok) return -1;
        }
        pap_prev = pap;
        if (COARSE && fabs(pap) < 1e-300) return (int)iter;
        stamp_it<TIMED>(a, iter, 1);
        const double alpha = rv / pap;
        // r += alpha A p; <r, z(r)>; |r|_inf against the stop; edge rows out
        c.step++;
        tm_stored();
        double rr = 0.0;
        bool above = false;
#pragma unroll 1
        for (int m0 = 0; m0 < units; m0 += kBatch) {
            Cell r[kBatch], ap[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                tm_load(ap[q], tap + 4 * min(m0 + q, units - 1));
                tm_load(r[q], tr + 4 * min(m0 + q, units - 1));
            }
            tm_loaded(ap);
            tm_loaded(r);
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                const int m = m0 + q;
                double2 rm = pair_of(r[q]);
                const double2 av = pair_of(ap[q]);
                rm.x = rm.x + alpha * av.x;
                rm.y = rm.y + alpha * av.y;
                if (m < units) tm_store(tr + 4 * m, rm);
                if (m < p.cnt) {
                    publish(a, p, m, rm, c.step);
                    rr += rz_term<KIND>(rm.x);
                    rr += rz_term<KIND>(rm.y);
                    above = above || fabs(rm.x) > stop || fabs(rm.y) > stop;
                }
                __syncwarp();
            }
        }
        stamp_it<TIMED>(a, iter, 2);
        // x += alpha p, which nothing waits for: done while the sum and the halo travel
        auto advance_x = [&]() {
            if (xg == nullptr) {
#pragma unroll 1
                for (int m0 = 0; m0 < units; m0 += kBatch) {
                    Cell xt[kBatch];
                    double2 pc[kBatch];
#pragma unroll
                    for (int q = 0; q < kBatch; q++) {
                        tm_load(xt[q], tx + 4 * min(m0 + q, units - 1));
                        pc[q] = ld2(P + p.o0 + min(m0 + q, units - 1) * p.pitch);
                    }
                    tm_loaded(xt);
#pragma unroll
                    for (int q = 0; q < kBatch; q++) {
                        double2 xv = pair_of(xt[q]);
                        xv.x = xv.x + alpha * pc[q].x;
                        xv.y = xv.y + alpha * pc[q].y;
                        if (m0 + q < units) tm_store(tx + 4 * (m0 + q), xv);
                    }
                }
                return;
            }
            constexpr int NB = 4;  // loads from L2 in flight
#pragma unroll 1
            for (int m0 = 0; m0 < p.cnt; m0 += NB) {
                double2 xv[NB];
#pragma unroll
                for (int q = 0; q < NB; q++)
                    if (m0 + q < p.cnt) xv[q] = ld2(xg + (m0 + q) * p.n2);
#pragma unroll
                for (int q = 0; q < NB; q++) {
                    if (m0 + q >= p.cnt) continue;
                    const double2 pc = ld2(P + p.o0 + (m0 + q) * p.pitch);
                    xv[q].x = xv[q].x + alpha * pc.x;
                    xv[q].y = xv[q].y + alpha * pc.y;
                    st2(xg + (m0 + q) * p.n2, xv[q]);
                }
            }
            __syncwarp();
        };
        how = 1;
        if (fixed_point_ok(rr_prev)) {
            double v = rr;
            const bool any = block_total(v, above);
            Posted w{};
            if (threadIdx.x == 0) w = fast_sum_post(a, c.seq, v, rr_prev, any);
            __syncwarp();
            advance_x();
            if (threadIdx.x == 0) sh.flag[1] = fast_sum_wait(a, c.seq, w);
            receive_halo();
            __syncthreads();
            how = sh.flag[1];
            c.seq++;
            if (how == 0) {
                rr = sh.res[0];
                above = sh.res[1] != 0.0;
            }
        } else {
            advance_x();
            receive_halo();
            __syncthreads();
        }
        tm_stored();
        ok = how >= 0 && sh.flag[0] == 0;
        if (!ok) return -1;
        if (how == 1) {
            const Reduced d = slow_reduce(a, c.slow_seq++, rr, above ? 1.0 : 0.0);
            rr = d.sum;
            above = d.max != 0.0;
            ok = d.ok;
            if (!ok) return -1;
        }
        stamp_it<TIMED>(a, iter, 3);
        rr_prev = rr;
        if (!above) return COARSE ? (int)iter + 1 : (int)iter;
        const double rnv = KIND == PC_IMPLICIT ? -rr / 6.0 : rr;
        beta = rnv / rv;
        rv = rnv;
        iter++;
    }
    return COARSE ? (int)limit : -1;
}

// Set-up of one point: r = A x0 - b of the program and its start x0 (grid_lcg.c:100-149,
// verlet.c:31-71, 152-193, plcg.c:28-166). Out of line: it runs once per solve and its many
// loads would otherwise claim the iteration's registers.
template <bool PB>
__device__ __noinline__ double2 start_residual(const EngineArgs& e, int i, int j, int k) {
    const Coef cf{e.ex, e.ey, e.ez, e.dg, 0.0, 0.0};
    double x0;
    const Nb o = nb_of(e.n, i, j, k);
    double b, ax;
    if (e.prog == PROG_INIT_FIELD) {
        b = e.q[o.c] * e.c;
        x0 = 0.0;
        ax = 0.0;
    } else if (e.prog == PROG_LCG_UPDATE) {
        b = e.q[o.c] * e.c;
        x0 = e.phi_old[o.c];
        ax = apply_at<PB>(o, cf, [&](long q) { return e.phi_old[q]; });
    } else if (e.prog == PROG_MAZE_LCG) {
        b = apply_at<PB>(o, cf, [&](long q) { return 2 * e.phi_old[q] - e.phi_prev[q]; }) + e.c * e.q[o.c];
        x0 = e.y[o.c];
        ax = apply_at<PB>(o, cf, [&](long q) { return e.y[q]; });
    } else {
        b = e.b[o.c];
        x0 = e.x0[o.c];
        ax = apply_at<PB>(o, cf, [&](long q) { return e.x0[q]; });
    }
    return make_double2(ax + -1.0 * b, x0);
}

// Right-hand side of the multigrid programs at one point: c q, for MaZe A (2 phi - phi_prev) + c q
// (grid_multigrid.c:151-160, verlet.c:108-110).
template <bool PB>
__device__ __noinline__ double mg_rhs(const EngineArgs& e, int i, int j, int k) {
    const Coef cf{e.ex, e.ey, e.ez, e.dg, 0.0, 0.0};
    const Nb o = nb_of(e.n, i, j, k);
    if (e.prog == PROG_MG_UPDATE) return e.q[o.c] * e.c;
    return apply_at<PB>(o, cf, [&](long q) { return 2 * e.phi_old[q] - e.phi_prev[q]; }) + e.c * e.q[o.c];
}

// conj_grad and its callers. HL: pairs of a row per lane (1 up to n = 64, 2 up to 128).
template <bool PB, int KIND, int HL, bool TIMED>
__global__ void __launch_bounds__(kThreads, 1) resident_cg_kernel(const __grid_constant__ ResArgs a) {
    Shared& sh = shared_state();
    const EngineArgs& e = a.e;
    const int n = e.n, units = a.pairs;
    // finite values in the rows that are read for nothing
    for (int x = threadIdx.x; x < a.smem_doubles; x += kThreads) smem[x] = 0.0;
    __syncthreads();
    if (threadIdx.x == 0) {
        sh.flag[0] = sh.flag[1] = 0;
        sh.lo[0] = sh.lo[1] = sh.hi[0] = sh.hi[1] = 0;
    }
    const Patch p = make_patch(n, a.Pi, a.Pj, 0);
    Ctl c;
    c.step = a.step0;
    const uint32_t tm = tm_alloc(&sh.tmem);
    const uint32_t tr = tm_own(tm), tap = tr + 4 * units, tx = tap + 4 * units;
    const int prog = e.prog;
    // The grid the program leaves x in. It may be the one it starts from, so it only changes
    // after the grid-wide sum below, when every CTA has read the old values.
    double* xout = (prog == PROG_INIT_FIELD || prog == PROG_LCG_UPDATE) ? e.phi_new : prog == PROG_MAZE_LCG ? e.y : e.x;
    double* xg = a.x_tmem ? nullptr : xout + p.g0;
    Coef cf{e.ex, e.ey, e.ez, e.dg, 0.0, 0.0};
    if (PB) {
        cf.eb = e.ex[0];
        cf.db = e.dg[0];
    }

    stamp<TIMED>(a, 0);
    double acc = 0.0;
#pragma unroll 1
    for (int m = 0; m < units; m++) {
        const int i = p.i0 + p.li0 + m, j = p.j0 + p.lj, k = 2 * p.kk;
        double2 x0 = make_double2(0.0, 0.0), v = x0;
        if (m < p.cnt) {
            const double2 s0 = start_residual<PB>(e, i, j, k), s1 = start_residual<PB>(e, i, j, k + 1);
            v = make_double2(s0.x, s1.x);
            x0 = make_double2(s0.y, s1.y);
            if (xg != nullptr) st2(xg + m * p.n2, x0);
            if (KIND == PC_IMPLICIT) {
                acc += v.x * (v.x * (1.0 / 6.0));
                acc += v.y * (v.y * (1.0 / 6.0));
            } else {
                acc += rz_term<KIND>(v.x);
                acc += rz_term<KIND>(v.y);
            }
        }
        __syncwarp();
        tm_store(tr + 4 * m, v);
        if (xg == nullptr) tm_store(tx + 4 * m, x0);
    }
    tm_stored();
    stamp<TIMED>(a, 1);
    const Reduced start = slow_reduce(a, c.slow_seq++, acc, 0.0);
    stamp<TIMED>(a, 2);
    acc = start.sum;
    bool ok = start.ok;
    int result = -1;
    if (ok)
        result = iterate<PB, KIND, false, HL, TIMED>(a, c, p, units, smem + kStateDoubles, tr, tap, tx, xg, cf, KIND == PC_IMPLICIT ? -acc : acc, 0.0, e.tol,
                                          (long)n * n, ok);
    if (ok) {
#pragma unroll 1
        for (int m = 0; m < units; m++) {
            const int g = p.g0 + m * p.n2;
            Cell xt[1];
            double2 v = make_double2(0.0, 0.0);
            if (xg == nullptr) {
                tm_load(xt[0], tx + 4 * m);
                tm_loaded(xt);
                v = pair_of(xt[0]);
            } else if (m < p.cnt) {
                v = ld2(xg + m * p.n2);
            }
            if (m < p.cnt) {
                if (prog == PROG_MAZE_LCG) {  // phi = (2 phi - phi_prev) - y (verlet.c:46-65)
                    const double2 f = ld2(e.phi_old + g), fp = ld2(e.phi_prev + g);
                    st2(e.phi_new + g, make_double2((2 * f.x - fp.x) + -1.0 * v.x, (2 * f.y - fp.y) + -1.0 * v.y));
                } else if (prog == PROG_INIT_FIELD) {
                    st2(e.y + g, make_double2(0.0, 0.0));
                }
                if (xg == nullptr) st2(xout + g, v);
            }
            __syncwarp();
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        e.result[0] = result;
        e.result[1] = ok ? 0 : 1;
    }
    tm_free(tm);
}

// ------------------------------------------------------------------------------------
// The reference's two-level multigrid (library/src/multigrid.c:99-168, multigrid_pb.c:270-328)
// on the same patches, for n a multiple of 4: x in the shared plane, the right-hand side in
// tensor memory, red-black half-sweeps that exchange the edge rows' new values as iterate()
// exchanges r's, and the coarse grid (n/2) solved by iterate() on patches of its own. Only
// the residual before the restriction and the coarse correction pass through global memory,
// with a grid barrier each.
//
// Each function below makes its patch anew: kept in registers across the coarse solve the
// two patches spilled into it.
//
// Measured on one B200, us per V-cycle, before (engine.cu) and now: 64^3 609 / 271, 96^3 714 /
// 318, 128^3 843 / 392, Poisson-Boltzmann 96^3 819 / 399, 128^3 1019 / 631. 230 to 290 us of it are the 50 coarse
// iterations (4.6 us each at 32^3, 5.5 at 64^3: the latency of two sums and a halo trip), a
// half-sweep takes 2.1 us at 64^3 and 7 us at 128^3 (issue). Tried: the coarse rows of the
// correction staged in shared memory (prolong 13 instead of 10 us), the next points' PB
// coefficients loaded ahead (spills: 59 instead of 47 us for four sweeps at 96^3).
// ------------------------------------------------------------------------------------
template <bool PB>
__device__ __forceinline__ Coef fine_coef(const ResArgs& a) {
    const EngineArgs& e = a.e;
    return {e.ex, e.ey, e.ez, e.dg, PB ? e.ex[0] : 0.0, PB ? e.dg[0] : 0.0};
}

// The Poisson-Boltzmann coefficients around one point.
struct PointFaces {
    double exc, exm, eyc, eym, ezc, ezm, d;
};
__device__ __forceinline__ PointFaces point_faces(const Patch& p, const Coef& cf, int m, int e, bool bulk) {
    PointFaces f = {cf.eb, cf.eb, cf.eb, cf.eb, cf.eb, cf.eb, cf.db};
    if (!bulk) {
        const int q = m < p.cnt ? m : p.cnt > 0 ? p.cnt - 1 : 0, g = p.g0 + q * p.n2 + e, n = p.n;
        f.exc = cf.ex[g];
        f.eyc = cf.ey[g];
        f.ezc = cf.ez[g];
        f.d = cf.dg[g];
        f.exm = cf.ex[g + (p.i0 + p.li0 + q == 0 ? (n - 1) * p.n2 : -p.n2)];
        f.eym = cf.ey[g + (p.j0 + p.lj == 0 ? (n - 1) * n : -n)];
        f.ezm = cf.ez[g + (e == 0 && p.kk == 0 ? n - 1 : -1)];
    }
    return f;
}

// `sweeps` red-black iterations on the plane, its halo current before and after: the points
// with (i + j + k) even, then odd (multigrid.c:636-729, neighbours i-1, i+1, j-1, j+1, k-1,
// k+1; multigrid_pb.c:544-640, i+1, i-1, j+1, j-1, k+1, k-1).
//
// Of each pair one element belongs to the colour, and it alternates along the column. The
// other element of row m is the pair's inner k neighbour of unit m and, at the same time, the
// i neighbour of units m - 1 and m + 1: one load per row serves three, and a unit takes four
// shared-memory loads instead of seven. Two units' loads and sums run together.
template <bool PB, int HL>
__device__ __noinline__ bool smooth(const ResArgs& a, Ctl& ctl, uint32_t trhs, int sweeps) {
    Shared& sh = shared_state();
    const Patch p = make_patch(a.e.n, a.Pi, a.Pj, 0);
    const Coef cf = fine_coef<PB>(a);
    double* P = smem + kStateDoubles;
    const int n = p.n, units = a.pairs, wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nh = halo_rows(p);
    const unsigned bulk = PB ? sh.bulk[wid] : 0u;
    const bool side = p.lj == 0 || p.lj == p.bj - 1;
    u64 step = ctl.step;
#pragma unroll 1
    for (int half = 0; half < 2 * sweeps; half++) {
        const int colour = half & 1, e0 = (p.i0 + p.li0 + p.j0 + p.lj + colour) & 1;
        // the outer k neighbour's distance from the first element of the pair, by e
        const int out0 = p.kk == 0 ? n - 1 : -1, out1 = p.kk == p.h - 1 ? 2 - n : 2;
        step++;
        ulonglong2* mine = a.strips + strip(a, blockIdx.x, step, 0) + 2 * p.kk;
        // the elements that are not this colour's in rows m0 - 1 and m0
        double wm = P[p.o0 - p.pitch + e0], w0 = P[p.o0 + (e0 ^ 1)];
#pragma unroll 1
        for (int m0 = 0; m0 < units; m0 += 2) {
            const bool two = m0 + 1 < units;
            const int o = p.o0 + m0 * p.pitch, o1 = two ? o + p.pitch : o;
            Cell t[2];
            tm_load(t[0], trhs + 4 * m0);
            tm_load(t[1], trhs + 4 * (two ? m0 + 1 : m0));
            // rows m0 + 1 and m0 + 2
            const double w1 = P[o + p.pitch + e0], w2 = P[o1 + p.pitch + (e0 ^ 1)];
            const double k0 = P[o + (e0 ? out1 : out0)], k1 = P[o1 + (e0 ? out0 : out1)];
            const double jm0 = P[o - n + e0], jp0 = P[o + n + e0];
            const double jm1 = P[o1 - n + (e0 ^ 1)], jp1 = P[o1 + n + (e0 ^ 1)];
            tm_loaded(t);
            const double2 b0 = pair_of(t[0]), b1 = pair_of(t[1]);
            const double r0 = e0 ? b0.y : b0.x, r1 = e0 ? b1.x : b1.y;
            const double km0 = e0 ? w0 : k0, kp0 = e0 ? k0 : w0, km1 = e0 ? k1 : w1, kp1 = e0 ? w1 : k1;
            double v0, v1;
            if (!PB) {
                double s0 = wm + w1, s1 = w0 + w2;
                s0 = s0 + jm0;
                s1 = s1 + jm1;
                s0 = s0 + jp0;
                s1 = s1 + jp1;
                s0 = s0 + km0;
                s1 = s1 + km1;
                s0 = s0 + kp0;
                s1 = s1 + kp1;
                v0 = (r0 - s0) * (-1.0 / 6.0);
                v1 = (r1 - s1) * (-1.0 / 6.0);
            } else {
                const PointFaces f = point_faces(p, cf, m0, e0, (bulk >> m0) & 1u);
                const PointFaces g = point_faces(p, cf, m0 + 1, e0 ^ 1, (bulk >> (m0 + 1)) & 1u);
                double s0 = f.exc * w1 + f.exm * wm, s1 = g.exc * w2 + g.exm * w0;
                s0 = s0 + f.eyc * jp0;
                s1 = s1 + g.eyc * jp1;
                s0 = s0 + f.eym * jm0;
                s1 = s1 + g.eym * jm1;
                s0 = s0 + f.ezc * kp0;
                s1 = s1 + g.ezc * kp1;
                s0 = s0 + f.ezm * km0;
                s1 = s1 + g.ezm * km1;
                s0 = s0 - r0;
                s1 = s1 - r1;
                v0 = s0 / (f.d < 1e-14 ? 1e-14 : f.d);
                v1 = s1 / (g.d < 1e-14 ? 1e-14 : g.d);
            }
            wm = w1;
            w0 = w2;
            auto put = [&](int m, int e, double v) {
                if (m >= p.cnt) return;
                const int li = p.li0 + m;
                P[p.o0 + m * p.pitch + e] = v;
                if (!side && li != 0 && li != p.bi - 1) return;
                ulonglong2* d = mine + e;
                if (li == 0) st_pair(d + p.lj * n, v, step);
                if (li == p.bi - 1) st_pair(d + a.cap + p.lj * n, v, step);
                if (p.lj == 0) st_pair(d + 2 * a.cap + li * n, v, step);
                if (p.lj == p.bj - 1) st_pair(d + 3 * a.cap + li * n, v, step);
            };
            put(m0, e0, v0);
            if (two) put(m0 + 1, e0 ^ 1, v1);
            __syncwarp();
        }
        // the neighbours' edge rows, this colour's points; nobody reads this colour meanwhile
        constexpr int NR = 4 / HL;
#pragma unroll 1
        for (int y0 = wid; y0 < nh; y0 += NR * kWarps) {
            int src[4], dst[4];
            u64 x[4];
#pragma unroll
            for (int q = 0; q < NR; q++) {
                const int row = y0 + q * kWarps;
                const bool any = row < nh;
                const int at = any ? halo_source(a, p, row, step) : 0, to = any ? halo_at(p, row) : 0;
                const int e = halo_parity(p, row, colour);
#pragma unroll
                for (int t = 0; t < HL; t++) {
                    const int k = 2 * (lane + 32 * t) + e;
                    const bool on = any && lane + 32 * t < p.h;
                    src[q * HL + t] = on ? at + k : -1;
                    dst[q * HL + t] = to + k;
                }
            }
            if (!receive_values<4>(a, src, step, x)) sh.flag[0] = 1;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (src[q] >= 0) P[dst[q]] = __longlong_as_double(x[q]);
        }
        __syncthreads();
        if (sh.flag[0]) return false;
    }
    ctl.step = step;
    return true;
}

// rf = -(A x) + rhs into the grid (multigrid.c:113-116), or max |A x - rhs| (the check after
// each V-cycle, grid_multigrid.c:188-199).
template <bool PB>
__device__ __noinline__ double residual(const ResArgs& a, uint32_t trhs, bool store) {
    const Patch p = make_patch(a.e.n, a.Pi, a.Pj, 0);
    const Coef cf = fine_coef<PB>(a);
    const double* P = smem + kStateDoubles;
    const unsigned bulk = PB ? shared_state().bulk[threadIdx.x >> 5] : 0u;
    double top = 0.0;
    double2 im = ld2(P + p.o0 - p.pitch), pc = ld2(P + p.o0);
#pragma unroll 1
    for (int m = 0; m < a.pairs; m++) {
        Cell t[1];
        tm_load(t[0], trhs + 4 * m);
        const int o = p.o0 + m * p.pitch;
        const double2 ip = ld2(P + o + p.pitch);
        const Around s = around(p, P, o, pc);
        const double2 v = PB ? apply_pb(s, im, pc, ip, ((bulk >> m) & 1u) ? bulk_faces(cf) : load_faces(p, cf, m))
                             : apply_lap(s, im, pc, ip);
        __syncwarp();
        tm_loaded(t);
        const double2 b = pair_of(t[0]);
        if (m < p.cnt) {
            if (store) st2(a.e.rf + p.g0 + m * p.n2, make_double2(-v.x + 1.0 * b.x, -v.y + 1.0 * b.y));
            else top = fmax(top, fmax(fabs(v.x + -1.0 * b.x), fabs(v.y + -1.0 * b.y)));
        }
        __syncwarp();
        im = pc;
        pc = ip;
    }
    return top;
}

// 27-point full weighting of rf at coarse (I, J, K) and (I, J, K + 1), K even
// (multigrid.c:523-594): the nine rows' five values each, all loads before the sums.
__device__ __noinline__ double2 restrict_pair(const double* in, int n, int I, int J, int K) {
    const int i = 2 * I, j = 2 * J, k = 2 * K;
    const int gi[3] = {i * n * n, (i + 1 == n ? 0 : i + 1) * n * n, (i == 0 ? n - 1 : i - 1) * n * n};
    const int gj[3] = {j * n, (j + 1 == n ? 0 : j + 1) * n, (j == 0 ? n - 1 : j - 1) * n};
    const int km = k == 0 ? n - 1 : k - 1;
    double v[3][3][5];  // [i, i + 1, i - 1][j, j + 1, j - 1][k - 1 .. k + 3]
#pragma unroll
    for (int x = 0; x < 3; x++)
#pragma unroll
        for (int y = 0; y < 3; y++) {
            const double* row = in + gi[x] + gj[y];
            const double2 lo = __ldcg(reinterpret_cast<const double2*>(row + k));
            const double2 hi = __ldcg(reinterpret_cast<const double2*>(row + k + 2));
            v[x][y][0] = __ldcg(row + km);
            v[x][y][1] = lo.x;
            v[x][y][2] = lo.y;
            v[x][y][3] = hi.x;
            v[x][y][4] = hi.y;
        }
    auto weigh = [&](int c) {  // centre at value c
        double f = v[2][0][c] + v[1][0][c];
        f = f + v[0][2][c];
        f = f + v[0][1][c];
        f = f + v[0][0][c - 1];
        f = f + v[0][0][c + 1];
        double e = v[1][0][c - 1] + v[1][0][c + 1];
        e = e + v[2][0][c - 1];
        e = e + v[2][0][c + 1];
        e = e + v[1][2][c];
        e = e + v[1][1][c];
        e = e + v[2][2][c];
        e = e + v[2][1][c];
        e = e + v[0][2][c - 1];
        e = e + v[0][2][c + 1];
        e = e + v[0][1][c - 1];
        e = e + v[0][1][c + 1];
        double q = v[1][1][c - 1] + v[1][1][c + 1];
        q = q + v[1][2][c - 1];
        q = q + v[1][2][c + 1];
        q = q + v[2][1][c - 1];
        q = q + v[2][1][c + 1];
        q = q + v[2][2][c - 1];
        q = q + v[2][2][c + 1];
        double s = 8.0 * v[0][0][c] + 4.0 * f;
        s = s + 2.0 * e;
        s = s + q;
        return s * (1.0 / 64.0);
    };
    return make_double2(weigh(1), weigh(3));
}

// The coarse correction: A_c e = restriction of rf by CG from zero (50 iterations, relative
// 1e-5; implicit Jacobi for the Laplacian, none for PB), e into the coarse grid array.
template <bool PB>
__device__ __noinline__ bool coarse_solve(const ResArgs& a, Ctl& ctl, uint32_t tm) {
    constexpr int KIND = PB ? PC_NONE : PC_IMPLICIT;
    const EngineArgs& e = a.e;
    Ctl c = ctl;
    const int nc = e.n / 2, units = a.cpairs;
    const Patch p = make_patch(nc, a.cPi, a.cPj, 1);
    const uint32_t tap = tm + 4 * units, tx = tap + 4 * units;
    const Coef cf{e.cex, e.cey, e.cez, e.cdg, PB ? e.cex[0] : 0.0, PB ? e.cdg[0] : 0.0};
    double acc = 0.0, top = 0.0;
#pragma unroll 1
    for (int m = 0; m < units; m++) {
        double2 v = make_double2(0.0, 0.0);
        if (m < p.cnt) {
            const int I = p.i0 + p.li0 + m, J = p.j0 + p.lj, K = 2 * p.kk;
            const double2 b = restrict_pair(e.rf, e.n, I, J, K);
            v = make_double2(-1.0 * b.x, -1.0 * b.y);  // r = A 0 - b
            acc += KIND == PC_IMPLICIT ? v.x * (v.x * (1.0 / 6.0)) : v.x * v.x;
            acc += KIND == PC_IMPLICIT ? v.y * (v.y * (1.0 / 6.0)) : v.y * v.y;
            top = fmax(top, fmax(fabs(v.x), fabs(v.y)));
        }
        __syncwarp();
        tm_store(tm + 4 * m, v);
        tm_store(tx + 4 * m, make_double2(0.0, 0.0));
    }
    tm_stored();
    const Reduced start = slow_reduce(a, c.slow_seq++, acc, top);
    bool ok = start.ok;
    if (ok && start.max != 0.0)
        iterate<PB, KIND, true, 1, false>(a, c, p, units, smem + a.coarse_at, tm, tap, tx, nullptr, cf,
                                          KIND == PC_IMPLICIT ? -start.sum : start.sum, start.max, 1e-5, 50, ok);
#pragma unroll 1
    for (int m = 0; m < units; m++) {
        Cell t[1];
        tm_load(t[0], tx + 4 * m);
        tm_loaded(t);
        if (m < p.cnt) st2(e.ec + p.g0 + m * p.n2, pair_of(t[0]));
        __syncwarp();
    }
    ctl = c;
    return ok;
}

// x += P e on the plane, halo rows included (multigrid.c:393-463: trilinear, weights (1, 0) on
// even fine indices and (1/2, 1/2) on odd ones).
__device__ __noinline__ void prolong(const ResArgs& a) {
    const Patch p = make_patch(a.e.n, a.Pi, a.Pj, 0);
    double* P = smem + kStateDoubles;
    const int n = p.n, nc = n / 2, lane = threadIdx.x & 31, nh = halo_rows(p), rows = p.bi * p.bj;
#pragma unroll 1
    for (int y = threadIdx.x >> 5; y < rows + nh; y += kWarps) {
        int li, lj;
        if (y < rows) {
            li = y / p.bj;
            lj = y - li * p.bj;
        } else {
            const int r = halo_at(p, y - rows) / n;
            li = r / (p.bj + 2) - 1;
            lj = r - (li + 1) * (p.bj + 2) - 1;
        }
        int i = p.i0 + li, j = p.j0 + lj;
        i = i < 0 ? n - 1 : i == n ? 0 : i;
        j = j < 0 ? n - 1 : j == n ? 0 : j;
        const int i0 = i >> 1, i1 = i0 + 1 == nc ? 0 : i0 + 1, j0 = j >> 1, j1 = j0 + 1 == nc ? 0 : j0 + 1;
        const double wi = (i & 1) ? 0.5 : 1.0, wj = (j & 1) ? 0.5 : 1.0;
        const double* c00 = a.e.ec + (i0 * nc + j0) * nc;
        const double* c10 = a.e.ec + (i1 * nc + j0) * nc;
        const double* c01 = a.e.ec + (i0 * nc + j1) * nc;
        const double* c11 = a.e.ec + (i1 * nc + j1) * nc;
        double* row = P + ((li + 1) * (p.bj + 2) + lj + 1) * n;
#pragma unroll 1
        for (int kk = lane; kk < p.h; kk += 32) {
            const int k1 = kk + 1 == nc ? 0 : kk + 1;
            const bool oi = i & 1, oj = j & 1;
            // the eight weights of prolong_at; those that are zero are left out
            double e0 = __ldcg(c00 + kk) * wi * wj, o0 = e0 * 0.5, o1 = __ldcg(c00 + k1) * wi * wj * 0.5;
            double t10[2] = {0.0, 0.0}, t01[2] = {0.0, 0.0}, t11[2] = {0.0, 0.0};
            if (oi) {
                t10[0] = __ldcg(c10 + kk) * 0.5 * wj;
                t10[1] = __ldcg(c10 + k1) * 0.5 * wj * 0.5;
            }
            if (oj) {
                t01[0] = __ldcg(c01 + kk) * wi * 0.5;
                t01[1] = __ldcg(c01 + k1) * wi * 0.5 * 0.5;
            }
            if (oi && oj) {
                t11[0] = __ldcg(c11 + kk) * 0.5 * 0.5;
                t11[1] = __ldcg(c11 + k1) * 0.5 * 0.5 * 0.5;
            }
            double ev = e0 + t10[0];
            ev = ev + t01[0];
            ev = ev + t11[0];
            double od = o0 + t10[0] * 0.5;
            od = od + t01[0] * 0.5;
            od = od + t11[0] * 0.5;
            od = od + o1;
            od = od + t10[1];
            od = od + t01[1];
            od = od + t11[1];
            double2 x = ld2(row + 2 * kk);
            x.x = x.x + 1.0 * ev;
            x.y = x.y + 1.0 * od;
            st2(row + 2 * kk, x);
        }
    }
    __syncthreads();
}

// PROG_MG_UPDATE and PROG_MAZE_MG (grid_multigrid.c:110-212, verlet.c:86-149, 212-271):
// V-cycles until |A x - b|_inf <= tol, at most 1000.
template <bool PB, int HL>
__global__ void __launch_bounds__(kThreads, 1) resident_mg_kernel(const __grid_constant__ ResArgs a) {
    Shared& sh = shared_state();
    const EngineArgs& e = a.e;
    const int n = e.n, units = a.pairs;
    const bool maze = e.prog == PROG_MAZE_MG;
    for (int x = threadIdx.x; x < a.smem_doubles; x += kThreads) smem[x] = 0.0;
    __syncthreads();
    Ctl c;
    c.step = a.step0;
    uint32_t trhs;
    {
        const Patch p = make_patch(n, a.Pi, a.Pj, 0);
        trhs = tm_own(tm_alloc(&sh.tmem));
        // the start (the MaZe unknown y or the extrapolated field) on the patch and its halo
        double* P = smem + kStateDoubles;
        const int lane = threadIdx.x & 31, nh = halo_rows(p), rows = p.bi * p.bj;
#pragma unroll 1
        for (int y = threadIdx.x >> 5; y < rows + nh; y += kWarps) {
            int r = y < rows ? (y / p.bj + 1) * (p.bj + 2) + y % p.bj + 1 : halo_at(p, y - rows) / n;
            const int li = r / (p.bj + 2) - 1, lj = r - (li + 1) * (p.bj + 2) - 1;
            int i = p.i0 + li, j = p.j0 + lj;
            i = i < 0 ? n - 1 : i == n ? 0 : i;
            j = j < 0 ? n - 1 : j == n ? 0 : j;
            const int g = (i * n + j) * n;
            for (int k = lane; k < n; k += 32)
                P[r * n + k] = maze ? e.y[g + k] : 2 * e.phi_old[g + k] - e.phi_prev[g + k];
        }
        const Coef cf = fine_coef<PB>(a);
        const unsigned bulk = PB ? bulk_units(p, cf, units) : 0u;
        if (lane == 0) sh.bulk[threadIdx.x >> 5] = bulk;
#pragma unroll 1
        for (int m = 0; m < units; m++) {
            double2 b = make_double2(0.0, 0.0);
            if (m < p.cnt) {
                const int i = p.i0 + p.li0 + m, j = p.j0 + p.lj, k = 2 * p.kk;
                b.x = mg_rhs<PB>(e, i, j, k);
                b.y = mg_rhs<PB>(e, i, j, k + 1);
            }
            __syncwarp();
            tm_store(trhs + 4 * m, b);
        }
        tm_stored();
        __syncthreads();
    }
    const uint32_t tcoarse = trhs + 4 * units;
    bool ok = true;
    int result = -1;
    for (int it = 1; it <= 1000 && ok; it++) {
        const int sweeps = PB ? 4 : 3;
        ok = smooth<PB, HL>(a, c, trhs, sweeps);
        if (!ok) break;
        residual<PB>(a, trhs, true);
        ok = grid_sync(&a.head->bar);
        if (!ok) break;
        ok = coarse_solve<PB>(a, c, tcoarse);
        if (!ok) break;
        ok = grid_sync(&a.head->bar);
        if (!ok) break;
        prolong(a);
        ok = smooth<PB, HL>(a, c, trhs, sweeps);
        if (!ok) break;
        const Reduced d = slow_reduce(a, c.slow_seq++, 0.0, residual<PB>(a, trhs, false));
        ok = d.ok;
        if (ok && d.max <= e.tol) {
            result = it;
            break;
        }
    }
    if (ok) {
        const Patch p = make_patch(n, a.Pi, a.Pj, 0);
        const double* P = smem + kStateDoubles;
#pragma unroll 1
        for (int m = 0; m < p.cnt; m++) {
            const int g = p.g0 + m * p.n2;
            const double2 x = ld2(P + p.o0 + m * p.pitch);
            if (maze) {  // phi = (2 phi - phi_prev) - y
                const double2 f = ld2(e.phi_old + g), fp = ld2(e.phi_prev + g);
                st2(e.y + g, x);
                st2(e.phi_new + g, make_double2((2 * f.x - fp.x) + -1.0 * x.x, (2 * f.y - fp.y) + -1.0 * x.y));
            } else {
                st2(e.phi_new + g, x);
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        e.result[0] = result;
        e.result[1] = ok ? 0 : 1;
    }
    tm_free(sh.tmem);
}

// ------------------------------------------------------------------------------------
// Host: patches, sizes, launch.
// ------------------------------------------------------------------------------------
struct Plan {
    int Pi = 0, Pj = 0, bi = 0, bj = 0;
    int pairs = 0;        // point pairs of the busiest thread
    size_t plane = 0;     // doubles of the plane of p
    size_t smem = 0;
};
constexpr size_t kSmemBudget = 226 * 1024;
// Pairs per thread: tensor memory holds 32 of one vector, so r, A p and x up to 10 pairs,
// r and A p up to 16.
constexpr int kMaxPairs = 16, kMaxPairsX = 10;

// SMs of the current device, a B200's 148 where there is none (planners ask for sizes too).
int sm_count() {
    static thread_local int dev_of = -1, sms = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) {
        if (dev == dev_of) return sms;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) {
            dev_of = dev;
            return sms;
        }
    }
    (void)cudaGetLastError();
    return 148;
}

// The patches of an n^3 grid: the split of the n x n rows that leaves the fewest pairs to the
// busiest thread, then the fewest halo rows, among those whose plane fits; a patch row of
// pairs (bj n / 2) takes at most one CTA's threads. Pi = 0 for sizes that are not
// served (above 128 the plane of p does not fit).
Plan find_plan(int n, int sms) {
    Plan best;
    if (n < 16 || n % 2 || n > 128) return best;
    const int h = n / 2;
    for (int pi = 1; pi <= n && pi <= sms; pi++)
        for (int pj = 1; pj <= n && pi * pj <= sms; pj++) {
            Plan q;
            q.Pi = pi;
            q.Pj = pj;
            q.bi = (n + pi - 1) / pi;
            q.bj = (n + pj - 1) / pj;
            if (q.bj * h > kThreads) continue;
            // patches are bi or bi - 1 rows by bj or bj - 1: the largest share over the four
            for (int bj = n / pj; bj <= q.bj; bj++) {
                const int S = kThreads / (bj * h), SL = (q.bi + S - 1) / S;
                if (SL > q.pairs) q.pairs = SL;
            }
            const int halo = 2 * (q.bi + q.bj);
            if (q.pairs > kMaxPairs || halo > kMaxHaloSteps * (kWarps - 1)) continue;
            // patches are bi or bi - 1 rows by bj or bj - 1: the largest plane over the four
            for (int bj = n / pj; bj <= q.bj; bj++)
                for (int bi = n / pi; bi <= q.bi; bi++)
                    q.plane = std::max(q.plane, (size_t)plane_rows(n, bi, bj, q.pairs) * (bj + 2) * n);
            q.smem = (q.plane + (size_t)halo * n + kStateDoubles) * sizeof(double);
            if (q.smem > kSmemBudget) continue;
            if (!best.Pi || q.pairs < best.pairs || (q.pairs == best.pairs && q.bi + q.bj < best.bi + best.bj)) best = q;
        }
    return best;
}
// The last plans are kept (a multigrid launch asks for two).
Plan make_plan(int n, int sms) {
    struct Entry {
        int n = 0, sms = 0;
        Plan plan;
    };
    static thread_local Entry kept[4];
    static thread_local int next = 0;
    for (const Entry& e : kept)
        if (e.n == n && e.sms == sms) return e.plan;
    Entry& e = kept[next++ & 3];
    e.n = n;
    e.sms = sms;
    e.plan = find_plan(n, sms);
    return e.plan;
}

template <int HL, bool TIMED>
const void* pick_kernel(bool pb, int kind) {
    if (pb) return (const void*)resident_cg_kernel<true, PC_IMPLICIT, HL, TIMED>;
    if (kind == PC_JACOBI) return (const void*)resident_cg_kernel<false, PC_JACOBI, HL, TIMED>;
    return (const void*)resident_cg_kernel<false, PC_IMPLICIT, HL, TIMED>;
}

std::atomic<u64> g_launches{0};

ResArgs common_args(const EngineArgs& e, const Plan& pl) {
    ResArgs a{};
    a.e = e;
    a.Pi = pl.Pi;
    a.Pj = pl.Pj;
    a.cap = std::max(pl.bi, pl.bj) * e.n;
    a.pairs = pl.pairs;
    a.step0 = ++g_launches << 24;
    a.head = static_cast<ResHeader*>(e.halo);
    a.strips = reinterpret_cast<ulonglong2*>(a.head + 1);
    return a;
}

void launch(const void* kernel, ResArgs& a, cudaStream_t stream) {
    const size_t smem = (size_t)a.smem_doubles * sizeof(double);
    MZB_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    MZB_CHECK(cudaMemsetAsync(a.head, 0, sizeof(ResHeader), stream));
    void* params[] = {&a};
    count_launch();
    MZB_CHECK(cudaLaunchCooperativeKernel(kernel, dim3(a.Pi * a.Pj), dim3(kThreads), params, smem, stream));
}

}  // namespace

size_t resident_halo_bytes(int n) {
    const Plan pl = make_plan(n, sm_count());
    if (!pl.Pi) return 0;
    const size_t cap = (size_t)(pl.bi > pl.bj ? pl.bi : pl.bj) * n;
    return sizeof(ResHeader) + (size_t)pl.Pi * pl.Pj * 2 * 4 * cap * sizeof(ulonglong2);
}

bool resident_cg_launch(const EngineArgs& e, cudaStream_t stream) {
    if (e.halo == nullptr) return false;
    int kind = PC_IMPLICIT;
    if (e.prog == PROG_PCG || (e.prog == PROG_MAZE_LCG && !e.pb)) kind = e.precond;
    else if (e.prog != PROG_CG && e.prog != PROG_INIT_FIELD && e.prog != PROG_LCG_UPDATE && e.prog != PROG_MAZE_LCG)
        return false;
    if (kind != PC_IMPLICIT && kind != PC_JACOBI) return false;
    if ((uintptr_t)e.x & 15) return false;  // a caller's own buffer; x is written in pairs
    const Plan pl = make_plan(e.n, sm_count());
    if (!pl.Pi) return false;
    ResArgs a = common_args(e, pl);
    a.smem_doubles = (int)(pl.smem / sizeof(double));
    a.x_tmem = pl.pairs <= kMaxPairsX ? 1 : 0;
    const bool one = e.n <= 64, timed = e.stamps != nullptr;
    const void* kf = one ? (timed ? pick_kernel<1, true> : pick_kernel<1, false>)(e.pb, kind)
                         : (timed ? pick_kernel<2, true> : pick_kernel<2, false>)(e.pb, kind);
    launch(kf, a, stream);
    return true;
}

bool resident_mg_launch(const EngineArgs& e, cudaStream_t stream) {
    if (e.halo == nullptr || (e.prog != PROG_MG_UPDATE && e.prog != PROG_MAZE_MG) || e.n % 4) return false;
    const Plan pl = make_plan(e.n, sm_count());
    if (!pl.Pi) return false;
    const Plan cp = make_plan(e.n / 2, pl.Pi * pl.Pj);  // the fine grid's CTAs, some without a coarse patch
    if (!cp.Pi || 4 * pl.pairs + 12 * cp.pairs > 128) return false;
    ResArgs a = common_args(e, pl);
    a.cPi = cp.Pi;
    a.cPj = cp.Pj;
    a.cpairs = cp.pairs;
    a.coarse_at = kStateDoubles + (int)pl.plane;
    // the coarse plane and halo rows, and what a CTA without a patch reads for nothing
    const int coarse = std::max((int)(cp.smem / sizeof(double)) - kStateDoubles, (cp.pairs + 3) * e.n);
    a.smem_doubles = a.coarse_at + coarse;
    const int ccap = std::max(cp.bi, cp.bj) * (e.n / 2);
    if (a.smem_doubles * sizeof(double) > kSmemBudget || ccap > a.cap) return false;
    const bool one = e.n <= 64;
    launch(e.pb ? (one ? (const void*)resident_mg_kernel<true, 1> : (const void*)resident_mg_kernel<true, 2>)
                : (one ? (const void*)resident_mg_kernel<false, 1> : (const void*)resident_mg_kernel<false, 2>),
           a, stream);
    return true;
}

}  // namespace mzb
