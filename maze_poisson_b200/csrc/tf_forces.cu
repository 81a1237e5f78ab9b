// Shifted-force pair forces -- Tosi-Fumi (Born-Mayer-Huggins), Lennard-Jones and soft-core
// repulsion (reference: library/src/forces.c:112-337, parameters particles.c:181-295). The
// reference sums every potential over both orders of each pair and halves the energy;
// here each pair inside r_cut = L/2 is evaluated once and its force applied to both ions
// with opposite signs (for the soft-core potential this is the reference's own i < j
// loop with Newton's third law).
//
// Compiled with --fmad=true: this kernel is bound by the FP64 pipe, and its results are
// already ulp-level (exp and inverse powers) rather than bit-level equal to the
// reference, which uses glibc exp/pow.
//
// Layout. Ions are sorted by linked cell (particles.cu), cut into blocks of 32 and the
// blocks into super-blocks of SB blocks. A CTA of 8 warps takes one super-block pair
// (SI, SJ) of a half shell (SJ = SI + d, d = 0 .. nsb/2, the middle distance only once). A
// warp holds two neighbouring I blocks, one ion of each per lane with its force in registers;
// the 16 / SB warps of an I pair split the J blocks of SJ, then the 32 steps of a block, among
// them. In step s lane l pairs its two ions with ion (l + s) mod 32 of the J block: two
// independent chains that share one load of the partner and one update of its reaction, kept
// in a warp-private shared array (structure of arrays, conflict-free) without atomics, with a
// __syncwarp per step. SB is the largest of 8, 4, 2 that still gives kTfMinCtas CTAs
// (tf_plan): with SB = 8 throughout, 250 ions were one CTA and 2000 ions 36.
// On the diagonal super-tile each unordered block pair is taken once (and each pair inside a
// block once: steps 1 .. 15 and half of step 16). A tile whose bounding boxes are farther
// apart than r_cut (minimum image, 1e-9 relative margin) is left out; pruning is off when a
// coordinate lies outside [0, L). A step in which no lane's pair lies inside r_cut skips the
// pair terms (a warp vote).
//
// Cost. At 16000 ions the kernel was bound by shared-memory wavefronts (68 %, FP64 pipe 49 %,
// issue 60 %): a pair loaded its partner, seven constants and the reaction, 34 wavefronts for
// 40 FP64 instructions, and a 64-bit load costs an SM four times what an FP64 instruction
// does. So one J ion serves two I ions, a pair beyond the exponential's range reads four
// constants in two loads, and nothing goes through the conversion pipe: the nearest image by
// adding and subtracting 1.5 2^52, 1/r from the hardware's FP64 approximation and two
// Newton-Raphson steps. Pairs that are not taken read a row of zeros instead of being
// selected out, and the exponential's branch follows both ions' other terms. At 16000 ions TF
// 659 -> 559 us, LJ 569 -> 486 us: 90 instructions, 40 of them FP64, for each of the N (N - 1) / 2
// pairs (123 instructions before), FP64 pipe 62 %, issue 61 %; what is left is the latency of
// 16 warps of two chains and the CTA's slowest warp.
//
// Determinism. Registers and warp arrays accumulate in step order; the warps' partials are
// summed in warp order; each ion's force is the sum of its super-tile partials in a
// fixed order (k_tf_gather over a host-built list), the energy the sum of the CTAs'
// energies in CTA order.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "particles.cuh"

namespace mzb {

constexpr int kTfSbMax = 8;                  // blocks of 32 ions per super-block, at most
constexpr int kTfWarps = 8;
constexpr int kTfThreads = kTfWarps * 32;
constexpr int kTfResident = 2;  // CTAs per SM
// CTAs below which smaller super-blocks pay: two waves of kTfResident on 148 SMs. SB = 8 / 4 / 2
// at 7600 ions 187 / 163 / 222 us, at 16000 ions 548 / 577 / - us; SB = 4 / 2 at 4394 ions
// 71 / 85 us. TF at 64 / 250 / 1024 / 2278 / 4394 / 7600 ions, SB = 8 throughout before:
// 20 / 54 / 101 / 100 / 138 / 230 us, now 10 / 10 / 10 / 32 / 71 / 163 us.
constexpr int kTfMinCtas = 592;
// Pair-constant table in shared memory, up to 8 types: one row of kTfRow 16-byte slots per
// type pair (80 bytes: the rows of four type pairs lie on different banks), and after them a
// row of zeros, which pairs that are not taken read instead.
constexpr int kTfRow = kPairConsts / 2 + 1;
constexpr int kTfZero = 64 * kTfRow;
constexpr int kTfTab = 65 * kTfRow;
// J blocks one warp walks: SB / 2 I pairs share 8 warps
constexpr int tf_nj(int sb) { return sb == 8 ? 4 : 1; }
// shared memory: table, both super-blocks' positions, the warps' reaction arrays (one per J
// block the warp walks) and I forces, both super-blocks' types
constexpr size_t tf_smem(int sb) {
    return sizeof(double) * (2 * kTfTab + 2 * sb * 96 + kTfWarps * tf_nj(sb) * 96 + kTfWarps * 192 + sb * 32);
}
constexpr size_t kTfSmem = tf_smem(8);

// min-image gap along one axis between the interval [lo, hi] and the cell [c0, c0 + cl]
__device__ __forceinline__ double axis_gap(double lo, double hi, double c0, double cl, double L) {
    double best = 1e300;
#pragma unroll
    for (int s = -1; s <= 1; s++) {
        const double a = c0 + s * L, b = a + cl;
        const double g = fmax(0.0, fmax(a - hi, lo - b));
        best = fmin(best, g);
    }
    return best;
}

// Shifted-force pair force (times 1/r, to be multiplied by the separation) and energy from a
// row of the table, without the exponential of TF (pair_exp); zero for the row of zeros. TF rows are stored as {C, D}, {alpha, beta},
// {A, B}, {sigma, range of the exponential}, the others in the order of P.tab.
template <int POT>
__device__ __forceinline__ void pair_terms(const double2* t, double r2, double ir, double& fr, double& vm) {
    if (POT == POT_TF) {  // forces.c:112-186: the force is B A ex - 6 C / r^7 - 8 D / r^9 - alpha
        const double2 cd = t[0], ab = t[1];
        const double ir2 = ir * ir, ir6 = ir2 * ir2 * ir2, g = ab.x * ir;
        const double c6 = ir6 * cd.x, d8 = ir6 * (cd.y * ir2), s = c6 + d8;
        fr = fma(-6.0 * ir2, fma(1.0 / 3.0, d8, s), -g);  // -(6 c6 + 8 d8) / r^2 - alpha / r
        vm = fma(g, r2, ab.y) - s;
    } else if (POT == POT_LJ) {  // forces.c:199-271
        const double2 se = t[0], ab = t[1];
        const double s = se.x * ir, s2 = s * s, s6 = s2 * s2 * s2, s12 = s6 * s6, e4 = 4 * se.y, g = ab.x * ir;
        fr = fma(e4 * (12 * s12 - 6 * s6), ir * ir, -g);
        vm = fma(e4, s12 - s6, fma(g, r2, ab.y));
    } else {  // forces.c:283-337
        const double2 nd = t[0], ba = t[1];
        const double p = ba.x * pow(nd.y * ir, nd.x), g = ba.y * ir;
        fr = fma(nd.x * p, ir * ir, -g);
        vm = p + fma(g, r2, t[2].x);
    }
}

// Bounding box of each block of 32 cell-ordered ions: [lo x, lo y, lo z, hi x, hi y, hi z].
__device__ __forceinline__ void k_tf_boxes_body(const ParticleDev& P, int bx) {
    const int lane = threadIdx.x & 31;
    const int b = (int)((bx * (long)blockDim.x + threadIdx.x) >> 5);
    const int nblk = (P.np + 31) / 32;
    if (b >= nblk) return;
    const int s = b * 32 + lane < P.np ? b * 32 + lane : b * 32;  // idle lanes mirror lane 0
    double lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; d++) lo[d] = hi[d] = P.spos[3 * s + d];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    if (lane < 3) {
        P.tf_box[6 * b + lane] = lo[lane];
        P.tf_box[6 * b + 3 + lane] = hi[lane];
    }
}
__global__ void k_tf_boxes(ParticleDev P) { k_tf_boxes_body(P, blockIdx.x); }

// 1/sqrt(x) for x in the range of squared pair distances (normal numbers): two Newton-Raphson
// steps for f(y) = 1/y^2 - x, y <- y + y (1/2 - x y^2 / 2), each of which squares the relative
// error, from the hardware's FP64 approximation (the PTX instruction rsqrt.approx.ftz.f64; its
// error is not counted on: the result is held to a few units in the last place by a test of
// pair forces against 80-bit arithmetic). k_tf at 16000 ions: 559 us; with an FP32 seed, which
// takes two conversions a pair, 578; with rsqrt() 594.
__device__ __forceinline__ double inv_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = 0.5 * x;
    y = fma(y, fma(-h * y, y, 0.5), y);
    return fma(y, fma(-h * y, y, 0.5), y);
}

// x minus the nearest multiple of L: adding and subtracting 1.5 2^52 rounds to an integer.
__device__ __forceinline__ double nearest_image(double x, double L, double invL) {
    constexpr double kRound = 6755399441055744.0;
    return fma(-L, fma(x, invL, kRound) - kRound, x);
}

struct PairSep {
    double dx, dy, dz, r2;
};
__device__ __forceinline__ PairSep pair_sep(double L, double invL, double xi, double yi, double zi, double xj, double yj,
                                            double zj) {
    PairSep p;
    p.dx = nearest_image(xi - xj, L, invL);
    p.dy = nearest_image(yi - yj, L, invL);
    p.dz = nearest_image(zi - zj, L, invL);
    p.r2 = p.dx * p.dx + p.dy * p.dy + p.dz * p.dz;
    return p;
}
// The exponential of TF: negligible beyond exp_limit for every type pair (tf_exp_r2_limit).
// Apart from pair_terms, so that no branch stands between the two ions' other terms.
__device__ __forceinline__ void pair_exp(const double2* t, double exp_limit, double r2, double ir, double& fr, double& vm) {
    if (r2 < exp_limit) {
        const double2 e = t[2];
        const double ex = e.x * exp(e.y * (t[3].x - r2 * ir));
        fr += e.y * ex * ir;
        vm += ex;
    }
}

template <int POT>
__device__ __forceinline__ void k_tf_body(const ParticleDev& P, int bx) {
    extern __shared__ __align__(16) double sm[];
    const int SB = P.tf_sb, NQ = SB * 32;
    // the warps of an I pair: jparts of its J blocks, sparts of a block's 32 steps
    const int ni = SB / 2, nj = tf_nj(SB), jparts = SB / nj, sparts = kTfWarps / ni / jparts;
    double2* tab = reinterpret_cast<double2*>(sm);      // [65][kTfRow]
    double* ipos = sm + 2 * kTfTab;                     // [SB][3][32]
    double* jpos = ipos + NQ * 3;                       // [SB][3][32]
    double* fjw = jpos + NQ * 3;                        // [8 warps][nj][3][32]
    double* fiw = fjw + kTfWarps * nj * 96;             // [8 warps][2][3][32]
    int* irow = reinterpret_cast<int*>(fiw + kTfWarps * 192);  // [SB][32]: first row of the ion's type
    int* jrow = irow + NQ;                              // [SB][32]: row of the ion's type within it
    const int st = bx;
    const int SI = P.tf_st[2 * st], SJ = P.tf_st[2 * st + 1];
    const bool diag = SI == SJ;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wi = w % ni, part = w / ni, jp = part % jparts, sp = part / jparts;
    const int t0 = jp * nj, s0 = sp * (32 / sparts), s1 = s0 + 32 / sparts;
    const int np = P.np, nblk = (np + 31) / 32, ntyp = P.ntyp;
    const double L = P.L, invL = 1.0 / L, rc2 = P.rcut * P.rcut;
    const int rc2hi = __double2hiint(rc2);
    const double prune2 = rc2 * (1.0 + 1e-9);
    const bool prune = P.flags[1] == 0;

    for (int x = threadIdx.x; x < ntyp * ntyp * kPairConsts; x += blockDim.x) {
        const int c = x % kPairConsts, src = POT == POT_TF ? (0x74106532 >> (4 * c)) & 15 : c;
        sm[(x / kPairConsts) * 2 * kTfRow + c] = P.tab[x - c + src];
    }
    if (threadIdx.x < 2 * kTfRow) sm[2 * kTfZero + threadIdx.x] = 0.0;
    bool absent = false;  // an ion of either super-block takes part in no pair (ParticleDev::stype)
    for (int q = threadIdx.x; q < NQ; q += blockDim.x) {
        const int gi = SI * NQ + q, gj = SJ * NQ + q, o = (q >> 5) * 96 + (q & 31);
        const bool vi = gi < np, vj = gj < np;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            ipos[o + 32 * d] = vi ? P.spos[3 * gi + d] : 0.0;
            jpos[o + 32 * d] = vj ? P.spos[3 * gj + d] : 0.0;
        }
        const int ti = vi ? P.stype[gi] : 0, tj = vj ? P.stype[gj] : 0;
        irow[q] = ti * ntyp * kTfRow;
        jrow[q] = tj * kTfRow;
        absent = absent || ti < 0 || tj < 0;
    }
    for (int x = threadIdx.x; x < kTfWarps * nj * 96; x += blockDim.x) fjw[x] = 0.0;
    absent = __syncthreads_or(absent);
    double exp_limit = 0.0;
    if (POT == POT_TF)
        for (int x = 0; x < ntyp * ntyp; x++) exp_limit = fmax(exp_limit, tab[x * kTfRow + 3].y);

    double fxa = 0.0, fya = 0.0, fza = 0.0, fxb = 0.0, fyb = 0.0, fzb = 0.0, e_acc = 0.0;
    const int ba = 2 * wi, bb = ba + 1, Ia = SI * SB + ba, Ib = Ia + 1;
    if (Ia < nblk) {
        const double *pa = ipos + ba * 96 + lane, *pb = pa + 96;
        const double xa = pa[0], ya = pa[32], za = pa[64], xb = pb[0], yb = pb[32], zb = pb[64];
        const int rowa = irow[ba * 32 + lane], rowb = irow[bb * 32 + lane];
        const bool va = Ia * 32 + lane < np && rowa >= 0, vb = Ib * 32 + lane < np && rowb >= 0;
        // whether block I (its index bi in SI) is paired with J block t (J), and how: 0 not, 1
        // every pair, 2 the block with itself
        auto mode_of = [&](int I, int bi, int J, int t) {
            if (I >= nblk || J >= nblk) return 0;
            if (diag) {
                const int d = (t - bi) & (SB - 1);
                if (d == 0) return 2;
                if (d > SB / 2 || (d == SB / 2 && bi >= SB / 2)) return 0;
            }
            if (prune) {
                const double *bI = P.tf_box + 6 * I, *bJ = P.tf_box + 6 * J;
                const double gx = axis_gap(bI[0], bI[3], bJ[0], bJ[3] - bJ[0], L);
                const double gy = axis_gap(bI[1], bI[4], bJ[1], bJ[4] - bJ[1], L);
                const double gz = axis_gap(bI[2], bI[5], bJ[2], bJ[5] - bJ[2], L);
                if (gx * gx + gy * gy + gz * gz > prune2) return 0;
            }
            return 1;
        };
        for (int t = t0; t < t0 + nj; t++) {
            const int J = SJ * SB + t;
            const int ma = mode_of(Ia, ba, J, t), mb = mode_of(Ib, bb, J, t);
            if ((ma | mb) == 0) continue;
            const double* jx = jpos + t * 96;
            const int* jr = jrow + t * 32;
            double* fj = fjw + (w * nj + t - t0) * 96;
            const int left = np - J * 32;  // ions of block J, if fewer than 32
            // all: every ion of the three blocks is there and every pair is taken
            auto steps = [&](auto all) {
                for (int s = s0; s < s1; s++) {
                    const int jj = (lane + s) & 31;
                    const double xj = jx[jj], yj = jx[32 + jj], zj = jx[64 + jj];
                    const int row = jr[jj];
                    const PairSep a = pair_sep(L, invL, xa, ya, za, xj, yj, zj);
                    const PairSep b = pair_sep(L, invL, xb, yb, zb, xj, yj, zj);
                    bool ina = a.r2 <= rc2, inb = b.r2 <= rc2;
                    if (!all.value) {
                        // a block with itself: each pair once
                        const bool half = s >= 1 && (s < 16 || (s == 16 && lane < 16)), vj = jj < left && row >= 0;
                        ina = ina && va && vj && (ma == 1 || (ma == 2 && half));
                        inb = inb && vb && vj && (mb == 1 || (mb == 2 && half));
                    }
                    // steps with no pair inside r_cut leave the terms out
                    if (!__any_sync(0xffffffffu, ina || inb)) continue;
                    // a pair that is not taken reads the row of zeros at a harmless distance (the
                    // upper word of r_cut^2): its force and energy come out as zero
                    const double2 *ra = tab + (ina ? rowa + row : kTfZero), *rb = tab + (inb ? rowb + row : kTfZero);
                    const double r2a = __hiloint2double(ina ? __double2hiint(a.r2) : rc2hi, __double2loint(a.r2));
                    const double r2b = __hiloint2double(inb ? __double2hiint(b.r2) : rc2hi, __double2loint(b.r2));
                    const double ira = inv_sqrt(r2a), irb = inv_sqrt(r2b);
                    double fa, ea, fb, eb;
                    pair_terms<POT>(ra, r2a, ira, fa, ea);
                    pair_terms<POT>(rb, r2b, irb, fb, eb);
                    if (POT == POT_TF) {
                        pair_exp(ra, exp_limit, r2a, ira, fa, ea);
                        pair_exp(rb, exp_limit, r2b, irb, fb, eb);
                    }
                    fxa = fma(fa, a.dx, fxa);
                    fya = fma(fa, a.dy, fya);
                    fza = fma(fa, a.dz, fza);
                    fxb = fma(fb, b.dx, fxb);
                    fyb = fma(fb, b.dy, fyb);
                    fzb = fma(fb, b.dz, fzb);
                    fj[jj] = fma(-fa, a.dx, fma(-fb, b.dx, fj[jj]));
                    fj[32 + jj] = fma(-fa, a.dy, fma(-fb, b.dy, fj[32 + jj]));
                    fj[64 + jj] = fma(-fa, a.dz, fma(-fb, b.dz, fj[64 + jj]));
                    e_acc += ea + eb;
                    __syncwarp();
                }
            };
            if (ma == 1 && mb == 1 && left >= 32 && Ib * 32 + 32 <= np && !absent)
                steps(std::true_type());
            else
                steps(std::false_type());
        }
    }
    // I and J sides: the warps' partials summed in warp order
    double* out = P.fpart + (size_t)st * 2 * SB * 96;
    double* fi = fiw + w * 192 + lane;
    fi[0] = fxa;
    fi[32] = fya;
    fi[64] = fza;
    fi[96] = fxb;
    fi[128] = fyb;
    fi[160] = fzb;
    __shared__ double esh[kTfWarps];
    e_acc = warp_sum(e_acc);
    if (lane == 0) esh[w] = e_acc;
    __syncthreads();
    for (int x = threadIdx.x; x < SB * 96; x += blockDim.x) {
        const int t = x / 96, jj = (x / 3) % 32, dd = x % 3;  // out layout [block][32][3]
        double v = 0.0;
        for (int q = t / 2; q < kTfWarps; q += ni) v += fiw[q * 192 + (t & 1) * 96 + dd * 32 + jj];
        out[x] = v;
        const int owner = t / nj, y = ((t - owner * nj) * 3 + dd) * 32 + jj;  // warp arrays [J block][3][32]
        v = 0.0;
        for (int q = 0; q < kTfWarps; q++)
            if ((q / ni) % jparts == owner) v += fjw[q * nj * 96 + y];
        out[SB * 96 + x] = v;
    }
    if (threadIdx.x == 0) {
        double e = 0.0;
        for (int q = 0; q < kTfWarps; q++) e += esh[q];
        P.epart[st] = e;
    }
}
template <int POT>
__global__ void __launch_bounds__(kTfThreads, kTfResident) k_tf(ParticleDev P) { k_tf_body<POT>(P, blockIdx.x); }

// Each ion's force: its super-tile partials in list order, scattered back to ion order. A CTA
// of four warps per block of 32 cell-ordered ions: each warp sums a quarter of the block's
// list for all 32 lanes (one ion each, their partials side by side), and the quarters are
// added in order. (One warp per block was a chain of up to 60 loads: 12 us where SB is small.)
constexpr int kTfGather = 4;
__device__ __forceinline__ void k_tf_gather_body(const ParticleDev& P, int b) {
    __shared__ double part[kTfGather][96];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double f[3] = {0.0, 0.0, 0.0};
    const int g0 = P.tf_gstart[b], len = P.tf_gstart[b + 1] - g0;
    const int e1 = g0 + len * (w + 1) / kTfGather;
#pragma unroll 8
    for (int e = g0 + len * w / kTfGather; e < e1; e++) {
        const int ent = P.tf_gent[e];
        const int st = ent >> 4, side = (ent >> 3) & 1, slot = ent & 7;
        const double* o = P.fpart + (((size_t)st * 2 + side) * P.tf_sb + slot) * 32 * 3 + lane * 3;
        f[0] += o[0];
        f[1] += o[1];
        f[2] += o[2];
    }
#pragma unroll
    for (int d = 0; d < 3; d++) part[w][d * 32 + lane] = f[d];
    __syncthreads();
    const int s = b * 32 + lane;
    if (w != 0 || s >= P.np) return;
    const int p = P.cell_ions[s];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double v = part[0][d * 32 + lane];
        for (int q = 1; q < kTfGather; q++) v += part[q][d * 32 + lane];
        P.fn[3 * p + d] = v;
    }
}
__global__ void k_tf_gather(ParticleDev P) { k_tf_gather_body(P, blockIdx.x); }

__device__ __forceinline__ void k_tf_energy_body(const ParticleDev& P, int bx) {
    double v[1] = {0.0};
    for (int x = threadIdx.x; x < P.tf_nst; x += blockDim.x) v[0] += P.epart[x];
    __shared__ double sh[4 * 32];
    block_sum<1>(v, sh);
    if (threadIdx.x == 0) P.red[1] = v[0];
}
__global__ void k_tf_energy(ParticleDev P) { k_tf_energy_body(P, blockIdx.x); }

TfShape tf_shape(int np) {
    TfShape t;
    t.nblk = (np + 31) / 32 > 0 ? (np + 31) / 32 : 1;
    t.sb = kTfSbMax;
    t.nsb = (t.nblk + t.sb - 1) / t.sb;
    while (t.sb > 2 && t.nsb * (t.nsb + 1) / 2 < kTfMinCtas) {
        t.sb /= 2;
        t.nsb = (t.nblk + t.sb - 1) / t.sb;
    }
    return t;
}

void tf_plan(ParticleDev& P) {
    dev_free(P.tf_st);
    dev_free(P.tf_gstart);
    dev_free(P.tf_gent);
    dev_free(P.tf_box);
    dev_free(P.fpart);
    dev_free(P.epart);
    const TfShape shape = tf_shape(P.np);
    const int nblk = shape.nblk, sb = shape.sb, nsb = shape.nsb;
    P.tf_sb = sb;
    std::vector<int> st;
    for (int si = 0; si < nsb; si++) {
        st.push_back(si);
        st.push_back(si);
        for (int d = 1; 2 * d <= nsb; d++) {
            if (2 * d == nsb && si >= nsb / 2) continue;  // the middle distance once
            st.push_back(si);
            st.push_back((si + d) % nsb);
        }
    }
    P.tf_nst = (int)st.size() / 2;
    std::vector<std::vector<int>> lists(nblk);
    for (int k = 0; k < P.tf_nst; k++)
        for (int side = 0; side < 2; side++)
            for (int slot = 0; slot < sb; slot++) {
                const int b = st[2 * k + side] * sb + slot;
                if (b < nblk) lists[b].push_back((k << 4) | (side << 3) | slot);
            }
    std::vector<int> gstart(nblk + 1, 0), gent;
    for (int b = 0; b < nblk; b++) {
        gent.insert(gent.end(), lists[b].begin(), lists[b].end());
        gstart[b + 1] = (int)gent.size();
    }
    auto up = [](void** d, const void* h, size_t bytes) {
        *d = dev_alloc(bytes);
        MZB_CHECK(cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice));
        MZB_CHECK(cudaStreamSynchronize(cudaStreamLegacy));  // landed before any later kernel
    };
    up((void**)&P.tf_st, st.data(), sizeof(int) * st.size());
    up((void**)&P.tf_gstart, gstart.data(), sizeof(int) * gstart.size());
    up((void**)&P.tf_gent, gent.data(), sizeof(int) * gent.size());
    P.tf_box = static_cast<double*>(dev_alloc(sizeof(double) * 6 * nblk));
    P.fpart = static_cast<double*>(dev_alloc(sizeof(double) * (size_t)P.tf_nst * 2 * sb * 32 * 3));
    P.epart = static_cast<double*>(dev_alloc(sizeof(double) * P.tf_nst));
    static unsigned long long attr_done = 0;  // devices whose kernels allow kTfSmem
    int dev = 0;
    MZB_CHECK(cudaGetDevice(&dev));
    if (!(attr_done >> (dev & 63) & 1ull)) {
        MZB_CHECK(cudaFuncSetAttribute(k_tf<POT_TF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        MZB_CHECK(cudaFuncSetAttribute(k_tf<POT_LJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        MZB_CHECK(cudaFuncSetAttribute(k_tf<POT_SC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        attr_done |= 1ull << (dev & 63);
    }
}

void tf_forces(ParticleDev& P, cudaStream_t s) {
    if (P.np == 0) {
        MZB_CHECK(cudaMemsetAsync(P.red + 1, 0, sizeof(double), s));
        return;
    }
    if (P.ntyp * P.ntyp > 64) fatal("pair forces: more than 8 particle types");
    if (!P.tf_st) fatal("pair forces: no plan (tf_plan)");
    const int nblk = (P.np + 31) / 32;
    count_launch();
    k_tf_boxes<<<(nblk * 32 + 255) / 256, 256, 0, s>>>(P);
    count_launch();
    if (P.pot == POT_LJ)
        k_tf<POT_LJ><<<P.tf_nst, kTfThreads, tf_smem(P.tf_sb), s>>>(P);
    else if (P.pot == POT_SC)
        k_tf<POT_SC><<<P.tf_nst, kTfThreads, tf_smem(P.tf_sb), s>>>(P);
    else
        k_tf<POT_TF><<<P.tf_nst, kTfThreads, tf_smem(P.tf_sb), s>>>(P);
    count_launch();
    k_tf_gather<<<nblk, kTfGather * 32, 0, s>>>(P);
    count_launch();
    k_tf_energy<<<1, 1024, 0, s>>>(P);
    MZB_CHECK(cudaGetLastError());
}

// The pair-force stages of a batched step over a replica table (particles.cuh): boxes,
// pair forces (one launch per potential present), gather, energy.
namespace {
__global__ void __launch_bounds__(256) kt_tfbox(const StageArgs* __restrict__ A, const int* __restrict__ start,
                                                int nsys) {
    table_run(A, start, nsys, [&](const StageArgs& a, int b) { k_tf_boxes_body(a.P, b); });
}
template <int POT>
__global__ void __launch_bounds__(kTfThreads, kTfResident) kt_tf(const StageArgs* __restrict__ A, const int* __restrict__ start,
                                                       int nsys) {
    table_run(A, start, nsys, [&](const StageArgs& a, int b) { k_tf_body<POT>(a.P, b); });
}
__global__ void __launch_bounds__(128) kt_tfg(const StageArgs* __restrict__ A, const int* __restrict__ start,
                                              int nsys) {
    table_run(A, start, nsys, [&](const StageArgs& a, int b) { k_tf_gather_body(a.P, b); });
}
__global__ void __launch_bounds__(1024) kt_tfe(const StageArgs* __restrict__ A, const int* __restrict__ start,
                                               int nsys) {
    table_run(A, start, nsys, [&](const StageArgs& a, int b) { k_tf_energy_body(a.P, b); });
}
void tf_tlaunch(const StageTable& t, int k, void (*kernel)(const StageArgs*, const int*, int), int threads,
                size_t smem, cudaStream_t s) {
    if (t.total[k] <= 0) return;
    count_launch();
    kernel<<<t.total[k], threads, smem, s>>>(t.args, t.start + k * (t.nsys + 1), t.nsys);
    MZB_CHECK(cudaGetLastError());
}
}  // namespace

void tf_stages(const StageTable& t, cudaStream_t s) {
    static unsigned long long attr_done = 0;  // devices whose table kernels allow kTfSmem
    int dev = 0;
    MZB_CHECK(cudaGetDevice(&dev));
    if (!(attr_done >> (dev & 63) & 1ull)) {
        MZB_CHECK(cudaFuncSetAttribute(kt_tf<POT_TF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        MZB_CHECK(cudaFuncSetAttribute(kt_tf<POT_LJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        MZB_CHECK(cudaFuncSetAttribute(kt_tf<POT_SC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        attr_done |= 1ull << (dev & 63);
    }
    tf_tlaunch(t, SK_TFBOX, kt_tfbox, 256, 0, s);
    tf_tlaunch(t, SK_TF_TF, kt_tf<POT_TF>, kTfThreads, kTfSmem, s);
    tf_tlaunch(t, SK_TF_LJ, kt_tf<POT_LJ>, kTfThreads, kTfSmem, s);
    tf_tlaunch(t, SK_TF_SC, kt_tf<POT_SC>, kTfThreads, kTfSmem, s);
    tf_tlaunch(t, SK_TFG, kt_tfg, 128, 0, s);
    tf_tlaunch(t, SK_TFE, kt_tfe, 1024, 0, s);
}

}  // namespace mzb
