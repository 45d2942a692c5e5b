// Single-pass MPDATA step (mpdata_order 2, FCT on or off): one launch per
// advect call for every species, each CTA one 56 x 22 column tile of one
// species marching up the column (or up a range of its levels).  Per level it
//
//   P0  recomputes the donor-cell pass q0 -> q1 two levels ahead on the tile
//       plus its halo (upwind_advection, adv_mpdata.f90:43-103), so q1 never
//       goes through HBM;
//   P1  forms the antidiffusive pseudo-velocities u2, v2, w2 with their
//       cross terms (mpdata_fluxes, adv_mpdata.f90:105-252), scaled by 0.5
//       and 0.5*dz (:378-380);
//   P2  forms the FCT limiter's per-cell bounds, in/out flux sums and beta
//       factors in x, y and z (flux_limiter, adv_mpdata.f90:254-350, in the
//       per-cell form of adv_mpdata_FCT_core.f90:47-116, first and last cells
//       of every line included), limits the vertical face below, finishes
//       the corrective donor-cell pass (adv_mpdata.f90:384) one level down
//       and stores it;
//   P3  limits the horizontal faces of the level below with the betas of the
//       two cells beside each.
//
// Data movement.  The level planes of q0 and of the per-step fields (U_m,
// V_m, W_m/dz, J*rho) arrive in shared memory by TMA (64 x 28 boxes of
// this GPU's own arrays, each CTA loading its own) one level ahead of use,
// completing on mbarriers; W_m, dz*J*rho and dz of the thread's own
// columns come by plain loads one level ahead.  Each thread owns an x-pair of
// columns in two adjacent rows and works on the pairs with packed f32x2
// arithmetic; x neighbours come by warp shuffles, y neighbours from the shared
// planes.
//
// Arithmetic (the template argument M).
//   A_EXACT  the reference's FP32 expressions in their order, every operation
//            rounded as the reference rounds it, so results equal the CPU
//            oracle bit for bit.  The work is packed and has no branch: a
//            quotient is formed from the hardware reciprocal approximation,
//            one Newton step (which makes the reciprocal correctly rounded)
//            and Markstein's residual correction (P. Markstein, "Computation
//            of elementary functions on the IBM RISC System/6000 processor",
//            IBM J. Res. Dev. 34, 1990), with the residual scaled by a power
//            of two so that it stays exact for subnormal operands.  The
//            conditions under which that equals IEEE division are checked
//            (see `worst` and the prep kernels' flags); a tile that does not
//            meet them is redone with A_IEEE before the CTA ends.
//   A_IEEE   the same expressions with the compiler's IEEE division: any
//            operand, including infinities and NaN.
//   A_FAST   the same scheme rewritten for throughput: reciprocals by the
//            hardware approximation, fused multiply-adds, reassociated pair
//            sums.  Its results differ from the reference in the last bits;
//            the tolerance is stated where it is tested.
//
// What bounds it, and why this shape.  Nothing here is near the HBM roofline
// (8 + 28/S bytes per cell-species): the kernel is bound by issue and latency.
// Two adjacent rows per thread (12 warps, 168 registers) load each operand
// once for both rows and form the faces between them once: 11.1
// warp-instructions per cell-species in A_FAST at 52 % of the issue slots,
// where one row per warp on 24 warps took 14.2 at 61 % and two rows 16 apart,
// reloaded for every face, on 16 warps 14.5 at 58 %.  A y face between two
// warps is formed once too and its flux passed through a plane.  The rings
// are deep enough for the donor pass to run two levels ahead, so a level needs
// two block barriers.  An iteration in the middle of the march is compiled
// without its level conditions: the few large blocks it becomes are what lets
// the scheduler interleave the rows (A_FAST 2.85 -> 2.36 ms at 512x512x40x12).
// The signs of a flux are split, not selected (3.26 -> 2.81 ms).  What runs beside the row warps (the halo rows, the
// TMA issue) is kept short, for the instruction cache (2.36 -> 2.32 ms).
// At 512x512x40x12: A_FAST 2.73 -> 2.32 ms per launch, A_EXACT 10.8 (IEEE
// division) -> 3.51 ms; at 187x301x33x5 A_FAST 0.338 -> 0.257 ms.
//
// Reference: src/physics/adv_mpdata.f90:43-413, adv_mpdata_FCT_core.f90:47-116.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "common.cuh"
#include "launch_split.h"
#include "mpdata_fused.cuh"
#include "tma.cuh"

namespace icar {

namespace op {
constexpr int PW = 64;               // plane width (floats): x from x0 to x0+63
constexpr int PH = 28;               // plane rows: y from j0-3 to j0+24
constexpr int NC = 11;               // row warps: warp w owns the output rows 2w+3 and 2w+4 of the plane
constexpr int NT = (NC + 1) * 32;    // the last warp takes the halo rows 1, 2 and 25, 26
constexpr int TX = PW - 8;           // 56 output columns of an inner column tile: plane x 4..59
constexpr int TY = PH - 6;           // 22 output rows: plane y 3..24
static_assert(TY == 2 * NC, "two output rows per warp");
constexpr int YB = PH - 3;           // first of the halo rows above the output rows
constexpr int PLANE = PW * PH;
constexpr uint32_t PLANE_BYTES = PLANE * sizeof(float);
// Planes.  The fields of a level sit side by side in a ring of four levels
// (powers of two: a level's slot is one mask), so a level costs a thread one
// address and every field of it a constant offset from there.
constexpr int F_U = 0, F_V = 1, F_G = 2, F_WP = 3, F_Q1 = 4, N4 = 5;   // U_m, V_m, J*rho, W_m/dz, q1: t-1 .. t+2
constexpr int S_Q0 = 4 * N4;                        // q0, eight levels: t-1 .. t+4
constexpr int S_FV = S_Q0 + 8, S_FY = S_FV + 1;     // unlimited flux through the south faces of level t, limited v2 there of t-1
constexpr int S_BYI = S_FY + 1, S_BYO = S_BYI + 1;  // y-limiter betas
constexpr int NPLANES = S_BYO + 1;
constexpr size_t SMEM = (size_t)NPLANES * PLANE * sizeof(float) + 128;
constexpr uint64_t WAIT_NS = 2000000000ull;  // a TMA wait gives up after 2 s
constexpr int MAXS = 32;             // species per launch

// Column tiles.  An inner tile's plane keeps 4 halo columns on each side
// (56 output columns; the plane origin stays 16-byte aligned for TMA).  The
// first and last tiles of a row sit on the domain's edges, where there is
// nothing to read beyond the edge, so the first outputs the 60 columns from
// x = 0 and the last ends at the domain's last column: nx = 512 takes 9
// tiles where 56-column tiling takes 10.
__host__ __device__ inline int tiles_x(int nx) { return nx <= PW ? 1 : 2 + max(0, (nx - 120 + TX - 1) / TX); }

// Plane origin x0 and output columns [xlo, xhi) (plane coordinates) of
// column tile tx of ntx.
__device__ __forceinline__ void xtile(int nx, int tx, int ntx, int &x0, int &xlo, int &xhi)
{
    if (ntx == 1) {
        x0 = 0, xlo = 0, xhi = nx;
    } else if (tx == 0) {
        x0 = 0, xlo = 0, xhi = PW - 4;
    } else {
        const int start = PW - 4 + TX * (tx - 1);   // first output column
        if (tx < ntx - 1) {
            x0 = start - 4, xlo = 4, xhi = PW - 4;
        } else {
            x0 = (nx - PW + 3) & ~3;               // the plane reaches the last column (at most 3 beyond)
            xlo = start - x0, xhi = nx - x0;
        }
    }
}
}  // namespace op

// Kernel parameters.  The tensor maps (64 x 1 x 28 boxes over (x, z, y))
// live in a device table (cudaMalloc'd, so every 128-byte map is 64-byte
// aligned as TMA requires): q0maps[s] for the species inputs, fmaps[0..3]
// for U_m, V_m, W_m/dz and J*rho.
struct OnePassParams {
    const CUtensorMap *q0maps;
    const CUtensorMap *fmaps;
    float *out[op::MAXS];
    const float *Wm, *DJR, *dz;
    int *err;            // 1: a TMA wait gave up; 2: a TMA operand was misaligned (loads skipped)
    int *flags;          // what the prep kernel found in the winds and metrics (FLAG_*)
    Geo g;
    int nspecies;
    int tiles_x;
    unsigned whole;      // (tile, species) pairs that march whole columns
    int parts;           // level ranges of the others
    float nzero;         // -0.0f, not a compile-time constant (see opx::mul2_sep)
};

namespace opx {

enum Arith { A_FAST = 0, A_EXACT = 1, A_IEEE = 2 };
constexpr unsigned FULL = 0xffffffffu;
constexpr float S48 = 0x1p48f, R48 = 0x1p-48f, S51 = 0x1p51f, R51 = 0x1p-51f;
// Bound of the magnitudes A_EXACT accepts (q0, pseudo-velocities, results).
constexpr float EXACT_MAX = 0x1p40f;

// pair of plane f at dy rows from the position `at` addresses in plane 0
__device__ __forceinline__ float2 ld2(const float *at, int f, int dy = 0)
{
    return *reinterpret_cast<const float2 *>(at + f * op::PLANE + dy * op::PW);
}
__device__ __forceinline__ void st2(float *at, int f, float2 v, int dy = 0)
{
    *reinterpret_cast<float2 *>(at + f * op::PLANE + dy * op::PW) = v;
}
__device__ __forceinline__ float up(float v) { return __shfl_up_sync(FULL, v, 1); }     // lane-1's value
__device__ __forceinline__ float dn(float v) { return __shfl_down_sync(FULL, v, 1); }   // lane+1's value
// the pair shifted one cell left (x-1, x) / right (x+1, x+2)
__device__ __forceinline__ float2 lft(float2 v) { return make_float2(up(v.y), v.x); }
__device__ __forceinline__ float2 rgt(float2 v) { return make_float2(v.y, dn(v.x)); }

// Hardware reciprocal approximation, flushing subnormal operands and results.
// Every divisor is a metric term (J*rho, dz*J*rho and their face sums), a
// sum of tracer values plus 1e-10, or a flux sum plus 1e-15: none is
// subnormal or above 2^126 (A_EXACT's checks catch one that is), and the
// non-flushing form needs a multi-instruction subnormal handling around each
// reciprocal.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 rcp2(float2 b) { return make_float2(rcp_approx(b.x), rcp_approx(b.y)); }
__device__ __forceinline__ float2 div2x(float2 a, float2 b) { return make_float2(a.x / b.x, a.y / b.y); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 max2(float2 a, float2 b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
__device__ __forceinline__ float2 min2(float2 a, float2 b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }

// a*b rounded by itself: ptxas may contract a packed multiply into a packed
// add that consumes it, so a product that feeds an add directly is written
// as a fused multiply-add with a -0.0 the compiler cannot see.
__device__ __forceinline__ float2 mul2_sep(float2 a, float2 b, float2 nz) { return fma2(a, b, nz); }

// max(m, |a|, |b|), NaN if any is NaN
__device__ __forceinline__ void worst_of(float &m, float2 v)
{
    asm("max.NaN.abs.f32 %0, %0, %1, %2;\n" : "+f"(m) : "f"(v.x), "f"(v.y));
}

// ---- A_EXACT quotients -----------------------------------------------------
// Everything works on the negated reciprocal and yields the negated quotient,
// which spares the sign flips.  nrcp(b) = -RN(1/b): the approximation is good
// to an ulp, and one Newton step from there rounds correctly for every
// significand (tests/exact_quotient_check.cu checks them all).
__device__ __forceinline__ float2 nrcp(float2 b)
{
    const float2 r0 = make_float2(rcp_approx(-b.x), rcp_approx(-b.y));
    return fma2(r0, fma2(b, r0, splat2(1.0f)), r0);
}
// -(a*2^48)/b correctly rounded, for quotients that are normal numbers: the
// numerator is scaled first, so the residual A + b*nq is exact even for the
// smallest subnormal numerator.
__device__ __forceinline__ float2 nquot48(float2 a, float2 b)
{
    const float2 nr = nrcp(b);
    const float2 A = mul2(a, splat2(S48));
    const float2 nq = mul2(A, nr);
    return fma2(fma2(b, nq, A), nr, nq);
}
// A divisor that several quotients share, scaled by 2^K for the residual.
struct ExDiv {
    float2 bs, nrs, nr;   // b*2^K, -2^-K/b, -1/b
};
__device__ __forceinline__ ExDiv exdiv(float2 b, float s, float r)
{
    ExDiv d;
    d.nr = nrcp(b);
    d.bs = mul2(b, splat2(s));
    d.nrs = mul2(d.nr, splat2(r));
    return d;
}
// -(a/b) where the quotient may be subnormal: the trial quotient is unscaled
// and the residual scaled, so the last operation rounds once at the
// quotient's own granularity.  It is correct unless the quotient is
// subnormal and lies exactly halfway between two floats, which needs b to be
// an even integer other than a power of two (b = B*2^e with B odd and
// e <= 0 keeps every quotient at least 2^-25 ulp off a midpoint, more than
// the error of the product of residual and reciprocal).  `tie` says that
// such a divisor occurs (FLAG_TIE); then the halfway case is rounded to
// even by hand.
__device__ __forceinline__ float tie_even(float nq, float nq0, float rem, float bs)
{
    if (fabsf(nq0) < 0x1p-125f && fabsf(rem) == bs * 0x1p-75f * 0x1p-75f)
        return (__float_as_int(nq0) & 1) ? copysignf(nq0 - copysignf(0x1p-149f, rem), nq0) : nq0;
    return nq;
}
__device__ __forceinline__ float2 nquot(float2 a, const ExDiv &d, bool tie)
{
    const float2 nq0 = mul2(a, d.nr);
    const float2 rem = fma2(d.bs, nq0, mul2(a, splat2(S48)));
    float2 nq = fma2(rem, d.nrs, nq0);
    if (__builtin_expect(tie, 0)) nq = make_float2(tie_even(nq.x, nq0.x, rem.x, d.bs.x), tie_even(nq.y, nq0.y, rem.y, d.bs.y));
    return nq;
}

// ---- pair arithmetic of the variants -----------------------------------------
// A_IEEE: scalar operations, never contracted.  A_EXACT and A_FAST: packed
// (in A_EXACT, ml must not feed an add; mul2_sep does).
template <int M>
__device__ __forceinline__ float2 ad(float2 a, float2 b)
{
    if constexpr (M == A_IEEE) return add2x(a, b);
    else return add2(a, b);
}
template <int M>
__device__ __forceinline__ float2 sb(float2 a, float2 b)
{
    if constexpr (M == A_IEEE) return sub2x(a, b);
    else return sub2(a, b);
}
template <int M>
__device__ __forceinline__ float2 ml(float2 a, float2 b)
{
    if constexpr (M == A_IEEE) return mul2x(a, b);
    else return mul2(a, b);
}

// A face velocity as its two signed parts, doubled: U+|U| and U-|U| (A_IEEE: the
// velocity itself, in p).  Using both parts instead of selecting the upwind
// one spares a comparison and moves per face.
struct Split {
    float2 p, n;
};
template <int M>
__device__ __forceinline__ Split split(float2 U)
{
    if constexpr (M == A_IEEE) return {U, U};
    const float2 a = abs2(U);
    return {add2(U, a), sub2(U, a)};
}
// Donor-cell flux ((U+|U|)*l + (U-|U|)*r)/2 (adv_mpdata.f90:23-41).  One of the
// two products is zero, so fusing the other with the sum rounds as the
// reference does.  A_FAST leaves the flux doubled (half_of takes the factor
// into the reciprocal the flux divergence is multiplied with).
template <int M>
__device__ __forceinline__ float2 flux(float2 l, float2 r, Split s, float2 nz)
{
    if constexpr (M == A_IEEE) {
        const float2 a = abs2(s.p);
        return mul2x(add2x(mul2x(add2x(s.p, a), l), mul2x(sub2x(s.p, a), r)), splat2(0.5f));
    }
    const float2 f = fma2(s.p, l, mul2(s.n, r));
    if constexpr (M == A_EXACT) return mul2_sep(f, splat2(0.5f), nz);
    else return f;
}
__device__ __forceinline__ float2 half_of(float2 a) { return mul2(a, splat2(0.5f)); }
// A cell's y difference, the flux through its north face (l: the cell, r: the
// one north of it) less the one through its south face.  A_FAST fuses the
// subtraction.
template <int M>
__device__ __forceinline__ float2 north_less(float2 l, float2 r, Split s, float2 south, float2 nz)
{
    if constexpr (M == A_FAST) return fma2(s.p, l, fma2(s.n, r, neg2(south)));
    else return sb<M>(flux<M>(l, r, s, nz), south);
}
// The flux as the limiter uses it, doubled in A_EXACT and A_FAST (its sums are
// halved in the same operation that adds 1e-15).
template <int M>
__device__ __forceinline__ float2 lflux(float2 l, float2 r, float2 U, float2 nz)
{
    const Split s = split<M>(U);
    if constexpr (M == A_IEEE) return flux<M>(l, r, s, nz);
    else return fma2(s.p, l, mul2(s.n, r));
}

// FCT beta num/den (den > 0): min(1, num/den) as the reference uses it.
// A_IEEE returns a quotient >= 1 as 1 without dividing and 0 for num == 0.
__device__ __forceinline__ float beta_ieee(float num, float den)
{
    if (num >= den) return 1.0f;
    if (num == 0.0f) return 0.0f;
    return num / den;
}
// The limiter terms of a pair of cells in one direction from their bounds and
// the fluxes through their two faces (as lflux gives them).
template <int M>
__device__ __forceinline__ void betas(float2 qmax, float2 qmin, float2 qc, float2 fl, float2 fr, float2 &bin,
                                      float2 &bout)
{
    const float2 z = splat2(0.0f), e15 = splat2(1e-15f), one = splat2(1.0f);
    const float2 fin = sb<M>(max2(z, fl), min2(z, fr)), fout = sb<M>(max2(z, fr), min2(z, fl));
    const float2 a = sb<M>(qmax, qc), b = sb<M>(qc, qmin);
    if constexpr (M == A_IEEE) {
        const float2 di = add2x(fin, e15), dout = add2x(fout, e15);
        bin = make_float2(beta_ieee(a.x, di.x), beta_ieee(a.y, di.y));
        bout = make_float2(beta_ieee(b.x, dout.x), beta_ieee(b.y, dout.y));
    } else if constexpr (M == A_EXACT) {
        // never subnormal: a num below 2^-126*den would need values so small
        // that den is its 1e-15
        bin = min2(one, mul2(nquot48(a, fma2(fin, splat2(0.5f), e15)), splat2(-R48)));
        bout = min2(one, mul2(nquot48(b, fma2(fout, splat2(0.5f), e15)), splat2(-R48)));
    } else {
        bin = min2(one, mul2(a, rcp2(fma2(fin, splat2(0.5f), e15))));
        bout = min2(one, mul2(b, rcp2(fma2(fout, splat2(0.5f), e15))));
    }
}

// Limited face velocity (adv_mpdata_FCT_core.f90:103-115): times the factor of
// its sign, min(bin_r, bout_l) for u > 0, min(bin_l, bout_r) otherwise (betas
// are at most 1).  Twice the limited velocity rounds as the limited velocity
// does (where it is subnormal, its flux is too small to change a cell).
template <int M>
__device__ __forceinline__ Split limit(float2 u, float2 bin_r, float2 bout_l, float2 bin_l, float2 bout_r)
{
    if constexpr (M == A_IEEE) {
        auto one = [](float u, float br, float ol, float bl, float orr) {
            if (u > 0.0f) return fminf(fminf(1.0f, br), ol) * u;
            if (u < 0.0f) return fminf(fminf(1.0f, bl), orr) * u;
            return u;
        };
        const float2 w = make_float2(one(u.x, bin_r.x, bout_l.x, bin_l.x, bout_r.x),
                                     one(u.y, bin_r.y, bout_l.y, bin_l.y, bout_r.y));
        return {w, w};
    }
    const Split s = split<M>(u);
    return {mul2(s.p, min2(bin_r, bout_l)), mul2(s.n, min2(bin_l, bout_r))};
}
// A split velocity through a plane: as one value and back.
template <int M>
__device__ __forceinline__ float2 join(Split s)
{
    if constexpr (M == A_IEEE) return s.p;
    else return add2(s.p, s.n);   // one part is zero
}
template <int M>
__device__ __forceinline__ Split unjoin(float2 w)
{
    if constexpr (M == A_IEEE) return {w, w};
    const Split s = split<M>(w);
    return {half_of(s.p), half_of(s.n)};
}

// ---- pseudo-velocity of a face -------------------------------------------------
// |U|(1-|U|/(0.5*Gs)) (hi-lo)/(hi+lo+eps), minus a cross term
// 0.5*U*ev*eq/Gs per tangential direction, in the reference's order.
template <int M>
__device__ __forceinline__ float2 base_o(float2 U, float2 Gs, const ExDiv &d, float2 hi, float2 lo)
{
    const float2 a = abs2(U);
    if constexpr (M == A_IEEE) {
        const float2 v = mul2x(a, sub2x(splat2(1.0f), div2x(a, mul2x(splat2(0.5f), Gs))));
        return div2x(mul2x(v, sub2x(hi, lo)), add2x(add2x(hi, lo), splat2(1e-10f)));
    } else {
        // |U|/(0.5*Gs) = 2|U|/Gs; where it is too small for an exact residual,
        // one minus it is 1 either way
        const float2 a2 = add2(a, a);
        const float2 nq = mul2(a2, d.nr);
        const float2 nx = fma2(fma2(Gs, nq, a2), d.nr, nq);
        const float2 F = mul2(a, add2(splat2(1.0f), nx));
        const float2 den = add2(add2(hi, lo), splat2(1e-10f));
        // not subnormal for |U| >= 2^-80 or zero
        return mul2(nquot48(mul2(F, sub2(lo, hi)), den), splat2(R48));
    }
}
// ev = 0.25*S, eq = (((a-b)+c)-d)/(den4+1e-10)
template <int M>
__device__ __forceinline__ float2 cross_term(float2 U, float2 Gs, const ExDiv &d, float2 S, float2 a, float2 b, float2 c,
                                             float2 dd, float2 den4)
{
    const float2 den = ad<M>(den4, splat2(1e-10f));
    if constexpr (M == A_IEEE) {
        const float2 eq = div2x(sub2x(add2x(sub2x(a, b), c), dd), den);
        return neg2(div2x(mul2x(mul2x(mul2x(splat2(0.5f), U), mul2x(splat2(0.25f), S)), eq), Gs));
    } else {
        // eq48 = 2^48 eq (the numerator with its sign turned), then
        // U*S*eq48 = 2^51 times the reference's 0.5*U*(0.25*S)*eq, divided by
        // Gs with the 2^51 taken out by the scaled divisor.  Where the
        // reference's product is subnormal it has fewer bits than this one,
        // but the term is then below 2^-120 and cannot change the sum with a
        // base term of a face with |U| >= 2^-80 that moves anything.
        const float2 eq48 = nquot48(add2(sub2(sub2(b, a), c), dd), den);
        const float2 A = mul2(mul2(U, S), eq48);
        const float2 nq = mul2(A, d.nrs);
        return fma2(fma2(d.bs, nq, A), d.nrs, nq);   // minus the term
    }
}
template <int M>
__device__ __forceinline__ float2 sum4(float2 a, float2 b, float2 c, float2 d)
{
    return ad<M>(ad<M>(ad<M>(a, b), c), d);
}

}  // namespace opx

// One tile's march over output levels [ka, kb).  INT: the whole 64 x 28 plane
// lies inside the domain's interior (x in [1, nx-2], y in [1, ny-2]), so no
// cell of the tile meets a domain edge: the edge cases of the reference
// (boundary ring, first/last cells of the limiter lines, faces that do not
// exist) drop out at compile time.  Tiles that touch an edge take the general
// form.  bars: two mbarriers with no phase completed.  Returns false when a
// TMA wait gave up (the flag in p.err is then set and the CTA must stop).
// worst: the largest magnitude A_EXACT met (NaN if it met one).
//
// Iteration t does, between two block barriers each,
//   I1  the limited horizontal faces of level t-1 (P3), P0 of level t+2, P1 of
//       level t;
//   I2  P2 of level t, then the update of level t-1 and its store.
// A y face is formed once, by the row north of it, and its flux passed to the
// row south of it through a plane.  A march from ka > 0 starts two levels
// below it (the limited flux through the bottom of ka needs the z betas of
// ka-1 and the w2 below that); the horizontal terms are formed for the
// output levels only.
template <int M, bool FCT, bool INT>
__device__ __forceinline__ bool onepass_tile(float *sm, uint64_t *bars, const OnePassParams &p, int s, int x0, int xlo,
                                             int xhi, int j0, int ka, int kb, bool tie, float &worst)
{
    using namespace op;
    using namespace opx;
    constexpr int R = 2;   // rows per thread
    const Geo g = p.g;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int y0 = j0 - 3;
    // the warp index through a shuffle from lane 0, so that the compiler
    // treats every row condition below as warp-uniform (plain branches, no
    // reconvergence bookkeeping)
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int X = 2 * lane;
    const int ia = x0 + X, ib = ia + 1;   // global x of the pair
    const CUtensorMap *mq = p.q0maps + s;
    const CUtensorMap *mU = p.fmaps, *mV = p.fmaps + 1, *mW = p.fmaps + 2, *mG = p.fmaps + 3;
    const float2 zero2 = splat2(0.0f), nz2 = splat2(p.nzero);

    // levels: iterations t0..kb, limiter and faces up to tl, q1 up to l1
    const int t0 = max(ka - 2, 0), f0 = max(t0 - 1, 0);
    const int tl = min(kb, nz - 1), l1 = min(kb + 1, nz - 1), lq = min(kb + 2, nz - 1);

    // ---- TMA issue (elected thread only): the loads of iteration t, on
    // bars[(t - t0) & 1].  TMA operands must be aligned (map 64 B, destination
    // 128 B, barrier 8 B); misaligned ones are reported (flag 2) and the loads
    // skipped, so the CTA finishes instead of faulting.
    const bool aligned = (((uintptr_t)mq | (uintptr_t)p.fmaps) & 63u) == 0 && ((smem_u32(sm) & 127u) | (smem_u32(bars) & 7u)) == 0;
    auto load_q0 = [&](int l, uint64_t *bar) { tma_load_3d(sm + (S_Q0 + (l & 7)) * PLANE, mq, x0, l, y0, bar); };
    auto load_uvg = [&](int l, uint64_t *bar) {
        float *to = sm + (l & 3) * (N4 * PLANE);
        tma_load_3d(to + F_U * PLANE, mU, x0, l, y0, bar);
        tma_load_3d(to + F_V * PLANE, mV, x0, l, y0, bar);
        tma_load_3d(to + F_G * PLANE, mG, x0, l, y0, bar);
    };
    auto load_w = [&](int l, uint64_t *bar) { tma_load_3d(sm + ((l & 3) * N4 + F_WP) * PLANE, mW, x0, l, y0, bar); };
    auto issue = [&](int t) {
        uint64_t *bar = &bars[(t - t0) & 1];
        if (!aligned) {
            mbar_arrive_expect_tx(bar, 0);
            return;
        }
        const bool q = t + 3 <= lq, u = t + 2 <= l1, w = t + 1 <= tl;
        mbar_arrive_expect_tx(bar, ((q ? 1u : 0u) + (u ? 3u : 0u) + (w ? 1u : 0u)) * PLANE_BYTES);
        if (q) load_q0(t + 3, bar);
        if (u) load_uvg(t + 2, bar);
        if (w) load_w(t + 1, bar);
    };
    // the first iteration's: everything it and the donor pass before it read
    auto issue_first = [&]() {
        if (!aligned) {
            atomicExch(p.err, 2);
            mbar_arrive_expect_tx(bars, 0);
            return;
        }
        const int qb = min(t0 + 3, lq), ub = min(t0 + 2, l1), wb = min(t0 + 1, tl);
        mbar_arrive_expect_tx(bars, (uint32_t)(qb - f0 + 1 + 3 * (ub - t0 + 1) + (wb - t0 + 1)) * PLANE_BYTES);
        for (int l = f0; l <= qb; l++) load_q0(l, bars);
        for (int l = t0; l <= ub; l++) load_uvg(l, bars);
        for (int l = t0; l <= wb; l++) load_w(l, bars);
    };
    // bounded wait on the batch of iteration n, by every thread; a thread
    // whose wait gave up raises the flag and reports false (the CTA then
    // agrees at its next barrier to stop)
    auto wait_mine = [&](int n) {
        const bool mine = mbar_wait_bounded(&bars[n & 1], (uint32_t)(n >> 1) & 1u, WAIT_NS);
        if (!mine) atomicExch(p.err, 1);
        return mine;
    };
    // a wait gave up: wait (bounded) for the batch so no copy is left in
    // flight into this CTA's shared memory, then stop
    auto drain = [&](int n) {
        mbar_wait_bounded(&bars[n & 1], (uint32_t)(n >> 1) & 1u, WAIT_NS);
        return false;
    };
    if (threadIdx.x == 0) {
        tma_prefetch_map(mq);
        issue_first();
    }

    // ---- rows
    const bool halo = warp == NC;               // warp-uniform
    const int Y = halo ? 1 : 2 * warp + 3;      // first plane row
    const int j = y0 + Y;
    float *const own = sm + Y * PW + X, *const top = sm + YB * PW + X;   // top: the halo warp's upper rows
    auto at4 = [&](float *at, int l) { return at + (l & 3) * (N4 * PLANE); };
    auto atq = [&](float *at, int l) { return at + (S_Q0 + (l & 7)) * PLANE; };
    auto row_offset = [&](int jj) {   // of (ia, level 0, jj), clamped into the array (fewer than 2^32 elements)
        return (uint32_t)ix(g, max(min(ia, g.P - 2), 0), 0, max(min(jj, ny - 1), 0));
    };
    const uint32_t rowc[R] = {row_offset(j), row_offset(j + 1)};
    const uint32_t lstride = (uint32_t)g.P;
    const bool inA = ia >= 0 && ia < nx, inB = ib >= 0 && ib < nx;
    auto jin = [&](int jr) { return INT || (jr >= 0 && jr < ny); };
    auto jint = [&](int jr) { return INT || (jr > 0 && jr < ny - 1); };
    // the pair's columns that this tile stores (rows start on 16-byte
    // boundaries and ia is even: the pair is 8-byte aligned)
    const bool sta = (INT || inA) && X >= xlo && X < xhi, stb = (INT || inB) && X + 1 >= xlo && X + 1 < xhi;
    float *const outs = p.out[s];
    auto ldcol = [&](const float *src, uint32_t row, int lev) -> float2 {
        return *reinterpret_cast<const float2 *>(src + (row + (uint32_t)lev * lstride));
    };

    // ---- P0: donor-cell pass at level L on two rows (at: the first one's
    // position, jr its global row) into the q1 plane of L.  wtop = W_m(L), djr =
    // dz*J*rho at L; v: on entry the flux through the bottom of L (the one
    // through the top of L-1), on return the flux through its top.
    auto donor = [&](int L, float *at, int jr, const float2 (&wtop)[R], const float2 (&djr)[R], float2 (&v)[R], float2 (&q1)[R]) {
        const float *Q = atq(at, L), *Qn = atq(at, L + 1), *F = at4(at, L);
        const float2 c[R + 2] = {ld2(Q, 0, -1), ld2(Q, 0), ld2(Q, 0, 1), ld2(Q, 0, 2)};
        float2 south = flux<M>(c[0], c[1], split<M>(ld2(F, F_V)), nz2);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float2 cc = c[r + 1];
            if constexpr (M == A_EXACT) worst_of(worst, cc);
            // a cell's east face is the next cell's west face: same operands,
            // same value, so it is formed once and passed along by a shuffle
            const float2 fw = flux<M>(lft(cc), cc, split<M>(ld2(F, F_U, r)), nz2), fe = rgt(fw);
            const Split vn = split<M>(ld2(F, F_V, r + 1));
            const float2 hd = ad<M>(sb<M>(fe, fw), north_less<M>(cc, c[r + 2], vn, south, nz2));
            if (r + 1 < R) south = flux<M>(cc, c[r + 2], vn, nz2);
            const float2 G = ld2(F, F_G, r);
            float2 vd;
            if (L < nz - 1) {
                const float2 vt = flux<M>(cc, ld2(Qn, 0, r), split<M>(wtop[r]), nz2);
                vd = sb<M>(vt, v[r]);
                v[r] = vt;
            } else if constexpr (M == A_FAST) {   // the model top: q times the face's W_m
                vd = fma2(cc, add2(wtop[r], wtop[r]), neg2(v[r]));
            } else if constexpr (M == A_EXACT) {
                vd = sub2(mul2_sep(cc, wtop[r], nz2), v[r]);
            } else {
                vd = sub2x(mul2x(cc, wtop[r]), v[r]);
            }
            float2 val;
            if constexpr (M == A_IEEE) {
                val = sub2x(sub2x(cc, div2x(hd, G)), div2x(vd, djr[r]));
            } else if constexpr (M == A_EXACT) {
                val = add2(cc, nquot(hd, exdiv(G, S48, R48), tie));
                val = add2(val, nquot(vd, exdiv(djr[r], S48, R48), tie));
            } else {
                val = sub2(sub2(cc, mul2(hd, half_of(rcp2(G)))), mul2(vd, half_of(rcp2(djr[r]))));
            }
            if (!INT) {
                const int jj = jr + r;
                const bool rin = jj >= 0 && jj < ny, jring = jj == 0 || jj == ny - 1;
                val.x = !(inA && rin) ? 0.0f : ((jring || ia == 0 || ia == nx - 1) ? cc.x : val.x);
                val.y = !(inB && rin) ? 0.0f : ((jring || ib == 0 || ib == nx - 1) ? cc.y : val.y);
            }
            q1[r] = val;
        }
    };
    // the flux through the top of level L on a row, for a march (or a row)
    // that does not carry it
    auto top_flux = [&](int L, float *at, uint32_t row) -> float2 {
        return flux<M>(ld2(atq(at, L), 0), ld2(atq(at, L + 1), 0), split<M>(ldcol(p.Wm, row, L)), nz2);
    };
    // ---- P1: pseudo-velocities at level t ------------------------------------
    // y face: v2 on the south faces of a row.  qc, qs: q1(t) of the row and of
    // the one south of it; qu, qsu, qd, qsd: the same at t+1 and t-1; the wind
    // and metric operands likewise.  The unlimited flux goes to its plane.
    auto face_y = [&](auto st, int t, int jr, float2 qc, float2 qs, float2 qu, float2 qsu, float2 qd, float2 qsd, float2 Vt,
                      float2 Gc, float2 Gst, float2 Ut, float2 Us, float2 Wt, float2 Wd, float2 Wts, float2 Wds,
                      float2 &fv) -> float2 {
        const bool kint = decltype(st)::value || (t > 0 && t < nz - 1);
        const float2 Gs = ad<M>(Gc, Gst);
        const bool xa = INT || (ia > 0 && ia < nx - 1), xb = INT || (ib > 0 && ib < nx - 1);
        float2 val;
        if constexpr (M != A_FAST) {
            ExDiv d{};
            if constexpr (M == A_EXACT) d = exdiv(Gs, S51, R51);
            val = base_o<M>(Vt, Gs, d, qc, qs);
            {
                const float2 qcl = lft(qc), qcr = rgt(qc), qsl = lft(qs), qsr = rgt(qs);
                const float2 Utr = rgt(Ut), Usr = rgt(Us);
                const float2 cp = make_float2(qc.y, qcr.y), sp = make_float2(qs.y, qsr.y);   // x+1
                float2 ct = cross_term<M>(Vt, Gs, d, sum4<M>(make_float2(Ut.y, Utr.y), make_float2(Us.y, Usr.y), Ut, Us),
                                          sp, qcl, cp, qsl, sum4<M>(cp, sp, qcl, qsl));
                // no cross term on the domain's first and last columns
                if (!xa) ct.x = 0.0f;
                if (!xb) ct.y = 0.0f;
                val = ad<M>(val, ct);
            }
            if (kint)
                val = ad<M>(val, cross_term<M>(Vt, Gs, d, sum4<M>(Wt, Wd, Wts, Wds), qsu, qd, qu, qsd,
                                               sum4<M>(qsu, qd, qu, qsd)));
            if constexpr (M == A_EXACT) val = mul2_sep(val, splat2(0.5f), nz2);
            else val = mul2x(val, splat2(0.5f));
        } else {
            // the final 0.5 folded in: 0.5 |V| (1 - 2 |V| / Gs) = 0.5 |V| - V^2 / Gs, and each
            // cross term 0.25 V / Gs times the 4-face average (1/4 of the face sum) times eq
            const float2 rG = rcp2(Gs);
            const float2 F0 = sub2(mul2(splat2(0.5f), abs2(Vt)), mul2(mul2(Vt, Vt), rG));
            const float2 sq = add2(qc, qs);
            val = mul2(mul2(F0, sub2(qc, qs)), rcp2(add2(sq, splat2(1e-10f))));
            const float2 mc = mul2(splat2(-0.0625f), mul2(Vt, rG));
            // x cross term: the two rows' pair sums at x+1 and x-1, and U_m on the
            // cells' west and east faces in both rows, each formed from one shuffle
            const float2 yp = rgt(sq), ym = lft(sq);
            float2 eq = mul2(sub2(yp, ym), rcp2(add2(add2(yp, ym), splat2(1e-10f))));
            const float2 su = add2(Ut, Us);
            float2 ev = add2(su, rgt(su));
            // no cross term on the domain's first and last columns (their
            // shuffled neighbours may lie outside the plane)
            if (!xa) ev.x = eq.x = 0.0f;
            if (!xb) ev.y = eq.y = 0.0f;
            val = fma2(mul2(mc, ev), eq, val);
            if (kint) {
                const float2 zp = add2(qu, qsu), zm = add2(qd, qsd);
                const float2 eq2 = mul2(sub2(zp, zm), rcp2(add2(add2(zp, zm), splat2(1e-10f))));
                val = fma2(mul2(mc, add2(add2(Wt, Wd), add2(Wts, Wds))), eq2, val);
            }
        }
        if (!INT) {
            const bool fin = jr >= 1 && jr <= ny - 1;
            val.x = (fin && inA) ? val.x : 0.0f;
            val.y = (fin && inB) ? val.y : 0.0f;
        }
        if constexpr (M == A_EXACT) worst_of(worst, val);
        if constexpr (FCT) fv = lflux<M>(qs, qc, val, nz2);
        return val;
    };
    // the same for a row of the halo warp
    auto face_y_row = [&](auto st, int t, int yr, float2 &f) -> float2 {
        float *at = sm + yr * PW + X;
        const float *C = at4(at, t), *Up = at4(at, t + 1), *Dn = at4(at, t - 1);
        return face_y(st, t, y0 + yr, ld2(C, F_Q1), ld2(C, F_Q1, -1), ld2(Up, F_Q1), ld2(Up, F_Q1, -1), ld2(Dn, F_Q1),
                      ld2(Dn, F_Q1, -1), ld2(C, F_V), ld2(C, F_G), ld2(C, F_G, -1), ld2(C, F_U), ld2(C, F_U, -1),
                      ld2(C, F_WP), ld2(Dn, F_WP), ld2(C, F_WP, -1), ld2(Dn, F_WP, -1), f);
    };
    // x faces ia, ib (west faces of the pair)
    auto face_x = [&](auto st, int t, int jr, float2 qc, float2 qn, float2 qs, float2 qu, float2 qd, float2 Ut, float2 Gt,
                      float2 Vt, float2 Vtn, float2 Wt, float2 Wd) -> float2 {
        const bool kint = decltype(st)::value || (t > 0 && t < nz - 1);
        const float2 qcl = lft(qc), Gs = ad<M>(Gt, lft(Gt));
        float2 val;
        if constexpr (M != A_FAST) {
            ExDiv d{};
            if constexpr (M == A_EXACT) d = exdiv(Gs, S51, R51);
            val = base_o<M>(Ut, Gs, d, qc, qcl);
            if (jint(jr)) {
                const float2 qnl = lft(qn), qsl = lft(qs);
                val = ad<M>(val, cross_term<M>(Ut, Gs, d, sum4<M>(Vt, Vtn, lft(Vt), lft(Vtn)), qn, qs, qnl, qsl,
                                               sum4<M>(qn, qs, qnl, qsl)));
            }
            if (kint) {
                const float2 qul = lft(qu), qdl = lft(qd);
                val = ad<M>(val, cross_term<M>(Ut, Gs, d, sum4<M>(Wt, Wd, lft(Wt), lft(Wd)), qu, qd, qul, qdl,
                                               sum4<M>(qu, qd, qul, qdl)));
            }
            if constexpr (M == A_EXACT) val = mul2_sep(val, splat2(0.5f), nz2);
            else val = mul2x(val, splat2(0.5f));
        } else {
            const float2 rG = rcp2(Gs);
            const float2 F0 = sub2(mul2(splat2(0.5f), abs2(Ut)), mul2(mul2(Ut, Ut), rG));
            val = mul2(mul2(F0, sub2(qc, qcl)), rcp2(add2(add2(qc, qcl), splat2(1e-10f))));
            const float2 mc = mul2(splat2(-0.0625f), mul2(Ut, rG));
            if (jint(jr)) {
                const float2 sv = add2(Vt, Vtn);
                const float2 xp = add2(qn, lft(qn)), xm = add2(qs, lft(qs));
                const float2 eq = mul2(sub2(xp, xm), rcp2(add2(add2(xp, xm), splat2(1e-10f))));
                val = fma2(mul2(mc, add2(sv, lft(sv))), eq, val);
            }
            if (kint) {
                const float2 sw = add2(Wt, Wd);
                const float2 xp = add2(qu, lft(qu)), xm = add2(qd, lft(qd));
                const float2 eq = mul2(sub2(xp, xm), rcp2(add2(add2(xp, xm), splat2(1e-10f))));
                val = fma2(mul2(mc, add2(sw, lft(sw))), eq, val);
            }
        }
        if (!INT) {
            val.x = (jin(jr) && ia >= 1 && ia <= nx - 1) ? val.x : 0.0f;
            val.y = (jin(jr) && ib >= 1 && ib <= nx - 1) ? val.y : 0.0f;
        }
        if constexpr (M == A_EXACT) worst_of(worst, val);
        return val;
    };
    // z face at the top of a level below the last (columns inside the domain interior)
    auto face_z = [&](int jr, float2 dz, float2 qc, float2 qu, float2 qn, float2 qs, float2 qnu, float2 qsu, float2 Wt,
                      float2 Gt, float2 Gu, float2 Ut, float2 Uu, float2 Vt, float2 Vtn, float2 Vu, float2 Vun) -> float2 {
        const float2 Gs = ad<M>(Gu, Gt);
        float2 val;
        if constexpr (M != A_FAST) {
            ExDiv d{};
            if constexpr (M == A_EXACT) d = exdiv(Gs, S51, R51);
            val = base_o<M>(Wt, Gs, d, qu, qc);
            {
                const float2 qcl = lft(qc), qcr = rgt(qc), qul = lft(qu), qur = rgt(qu);
                const float2 Utr = rgt(Ut), Uur = rgt(Uu);
                const float2 cp = make_float2(qc.y, qcr.y), pp = make_float2(qu.y, qur.y);   // x+1
                val = ad<M>(val, cross_term<M>(Wt, Gs, d,
                                               sum4<M>(make_float2(Ut.y, Utr.y), make_float2(Uu.y, Uur.y), Ut, Uu), pp,
                                               qcl, cp, qul, sum4<M>(cp, pp, qcl, qul)));
            }
            val = ad<M>(val, cross_term<M>(Wt, Gs, d, sum4<M>(Vt, Vu, Vtn, Vun), qnu, qs, qn, qsu,
                                           sum4<M>(qn, qsu, qnu, qs)));
            if constexpr (M == A_EXACT) val = mul2_sep(mul2(val, splat2(0.5f)), dz, nz2);
            else val = mul2x(mul2x(val, splat2(0.5f)), dz);
        } else {
            const float2 rG = rcp2(Gs);
            const float2 F0 = sub2(mul2(splat2(0.5f), abs2(Wt)), mul2(mul2(Wt, Wt), rG));
            const float2 sq = add2(qc, qu);
            val = mul2(mul2(F0, sub2(qu, qc)), rcp2(add2(sq, splat2(1e-10f))));
            const float2 mc = mul2(splat2(-0.0625f), mul2(Wt, rG));
            const float2 zp = rgt(sq), zm = lft(sq);
            const float2 eq = mul2(sub2(zp, zm), rcp2(add2(add2(zp, zm), splat2(1e-10f))));
            const float2 su = add2(Ut, Uu);
            val = fma2(mul2(mc, add2(su, rgt(su))), eq, val);
            const float2 np = add2(qn, qnu), sp = add2(qs, qsu);
            const float2 eq2 = mul2(sub2(np, sp), rcp2(add2(add2(np, sp), splat2(1e-10f))));
            const float2 sv = add2(add2(Vt, Vu), add2(Vtn, Vun));
            val = fma2(mul2(mc, sv), eq2, val);
            val = mul2(val, dz);
        }
        if (!INT) {
            const bool jj = jr >= 1 && jr <= ny - 2;
            val.x = (jj && ia >= 1 && ia <= nx - 2) ? val.x : 0.0f;
            val.y = (jj && ib >= 1 && ib <= nx - 2) ? val.y : 0.0f;
        }
        if constexpr (M == A_EXACT) worst_of(worst, val);
        return val;
    };
    // y-line betas of a row at level t (its unlimited south flux from the own
    // value, its north one from the plane), stored for its neighbours too
    auto betas_y = [&](int jr, float *at, float2 qc, float2 q0c, float2 qs, float2 q0s, float2 qn, float2 q0n, float2 fl,
                       float2 &bi, float2 &bo) {
        float2 fr = ld2(at, S_FV, 1);
        float2 hs = max2(qs, q0s), ls = min2(qs, q0s), hn = max2(qn, q0n), ln = min2(qn, q0n);
        float2 hc = max2(qc, q0c), lc = min2(qc, q0c);
        if (!INT) {   // line ends (row-uniform), as in the x lines below
            if (jr == 0) { hs = hc; ls = lc; }
            if (jr == ny - 1) { hc = lc = hn = ln = qc; }
            if (jr == 0 || jr == ny - 1) fl = fr = zero2;
        }
        betas<M>(max2(max2(hs, hc), hn), min2(min2(ls, lc), ln), qc, fl, fr, bi, bo);
    };

    // ---- prologue: batch 0 landed -> q1 at levels t0 and t0+1 --------------
    // carried between iterations, per row: the donor pass's flux through the
    // top of the level it formed last (vt); level t's pseudo-velocities,
    // betas and vertical flux, and those of the level below that the z line
    // needs; the limited flux through the bottom of level t-1; the own-column
    // values loaded ahead
    float2 vt[R], n_wm[R], n_djr[R], n_dz[R], djr_m[R];
    float2 u2[R], v2[R], w2[R], w2b[R], fz[R], fzb[R], bxi[R], bxo[R], byi[R], byo[R], bzi[R], bzo[R], hx[R], fb[R], gm[R], fs = zero2;
#pragma unroll
    for (int r = 0; r < R; r++) {
        vt[r] = n_wm[r] = n_dz[r] = u2[r] = v2[r] = w2[r] = w2b[r] = fz[r] = fzb[r] = zero2;
        bxi[r] = bxo[r] = byi[r] = byo[r] = bzi[r] = bzo[r] = hx[r] = fb[r] = zero2;
        n_djr[r] = djr_m[r] = gm[r] = splat2(1.0f);
    }
    // The halo warp carries the donor pass's state for its two row pairs: the
    // lower pair's in vt, n_wm and n_djr, the upper pair's in these (which its
    // rows do not need otherwise).
    float2(&vt_b)[R] = u2, (&wm_b)[R] = bxi, (&djr_b)[R] = bxo;
    const uint32_t rowb[R] = {row_offset(y0 + YB), row_offset(y0 + YB + 1)};
    if (__syncthreads_and(wait_mine(0) ? 1 : 0) == 0) return drain(0);
    auto load_ahead = [&](int L) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            n_wm[r] = ldcol(p.Wm, rowc[r], L);
            n_djr[r] = ldcol(p.DJR, rowc[r], L);
        }
    };
    auto load_ahead_b = [&](int L) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            wm_b[r] = ldcol(p.Wm, rowb[r], L);
            djr_b[r] = ldcol(p.DJR, rowb[r], L);
        }
    };
    // (loops, with the two pairs' state swapped: the halo warp's code has to
    // fit the instruction cache beside the row warps')
    auto donor_halo = [&](int L) {
#pragma unroll 1
        for (int q = 0; q < 2; q++) {
            float *at = q == 0 ? own : top;
            float2 q1[R];
            donor(L, at, q == 0 ? j : y0 + YB, n_wm, n_djr, vt, q1);
#pragma unroll
            for (int r = 0; r < R; r++) {
                st2(at4(at, L), F_Q1, q1[r], r);
                const float2 a = vt[r], b = n_wm[r], c = n_djr[r];
                vt[r] = vt_b[r], n_wm[r] = wm_b[r], n_djr[r] = djr_b[r];
                vt_b[r] = a, wm_b[r] = b, djr_b[r] = c;
            }
            if constexpr (M == A_EXACT) worst_of(worst, ld2(atq(at, L), 0, q == 0 ? -1 : 2));   // the plane's end rows
        }
    };
    for (int L = t0; L <= min(t0 + 1, l1); L++) {
        load_ahead(L);
#pragma unroll
        for (int r = 0; r < R; r++)
            if (L == t0 && t0 > 0) vt[r] = top_flux(t0 - 1, own + r * PW, rowc[r]);
        if (halo) {
            load_ahead_b(L);
#pragma unroll
            for (int r = 0; r < R; r++)
                if (L == t0 && t0 > 0) vt_b[r] = top_flux(t0 - 1, top + r * PW, rowb[r]);
            donor_halo(L);
        } else {
            float2 q1[R];
            donor(L, own, j, n_wm, n_djr, vt, q1);
#pragma unroll
            for (int r = 0; r < R; r++) st2(at4(own, L), F_Q1, q1[r], r);
        }
    }
    if (t0 + 2 <= l1) {
        load_ahead(t0 + 2);
        if (halo) load_ahead_b(t0 + 2);
    }
#pragma unroll
    for (int r = 0; r < R; r++) n_dz[r] = ldcol(p.dz, rowc[r], t0);
    __syncthreads();   // q1 of t0 and t0+1 complete

    // ST: an iteration in the middle of a march, where every condition on the
    // level holds; it compiles to few large blocks, which the scheduler can
    // interleave.
    auto level = [&](auto st, const int t) -> bool {
        constexpr bool ST = decltype(st)::value;
        const int n = t - t0;
        const bool hor = ST || (t >= ka && t < kb);          // level t's horizontal terms are needed
        bool landed;
        if (!halo) {
            float2 vs = zero2;
            float *C = at4(own, t), *Up = at4(own, t + 1), *Dn = at4(own, t - 1);
            // ---- P3: limited west and south faces of level t-1 -----------------
            if (ST || t - 1 >= ka) {
                const float2 q[R + 1] = {ld2(Dn, F_Q1, -1), ld2(Dn, F_Q1), ld2(Dn, F_Q1, 1)};
                [[maybe_unused]] float2 bs = zero2, os = zero2;
                if constexpr (FCT) {
                    bs = ld2(own, S_BYI, -1);
                    os = ld2(own, S_BYO, -1);
                }
                float2 below = zero2;   // the first row's south flux
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float2 qc = q[r + 1], qcl = lft(qc);
                    Split u, v;
                    if constexpr (FCT) {
                        u = limit<M>(u2[r], bxi[r], lft(bxo[r]), lft(bxi[r]), bxo[r]);
                        v = limit<M>(v2[r], byi[r], os, bs, byo[r]);
                        bs = byi[r];
                        os = byo[r];
                    } else {
                        u = split<M>(u2[r]);
                        v = split<M>(v2[r]);
                    }
                    // east faces as the next cell's limited west faces
                    const float2 fw = flux<M>(qcl, qc, u, nz2), fn = flux<M>(q[r], qc, v, nz2);
                    hx[r] = sb<M>(rgt(fw), fw);
                    gm[r] = ld2(Dn, F_G, r);   // its plane is refilled after the next barrier
                    if (r == 0) {
                        below = fn;
                        vs = join<M>(v);
                    } else {   // the first row's divergence is complete
                        hx[0] = ad<M>(hx[0], north_less<M>(q[r], qc, v, below, nz2));
                        fs = fn;
                    }
                }
            }
            landed = wait_mine(n);
            // ---- P0: q1 at level t+2 ----------------------------------------
            float2 q1n[R], fv[R];
            if (ST || t + 2 <= l1) donor(t + 2, own, j, n_wm, n_djr, vt, q1n);
            // ---- P1: pseudo-velocities at level t -----------------------------
#pragma unroll
            for (int r = 0; r < R; r++) {
                w2b[r] = w2[r];
                fzb[r] = fz[r];
            }
            if (ST || t <= tl) {
                const float2 qc[R + 2] = {ld2(C, F_Q1, -1), ld2(C, F_Q1), ld2(C, F_Q1, 1), ld2(C, F_Q1, 2)};
                const float2 qu[R + 2] = {ld2(Up, F_Q1, -1), ld2(Up, F_Q1), ld2(Up, F_Q1, 1), ld2(Up, F_Q1, 2)};
                const float2 U[R + 1] = {ld2(C, F_U, -1), ld2(C, F_U), ld2(C, F_U, 1)};
                const float2 V[R + 1] = {ld2(C, F_V), ld2(C, F_V, 1), ld2(C, F_V, 2)};
                const float2 W[R + 1] = {ld2(C, F_WP, -1), ld2(C, F_WP), ld2(C, F_WP, 1)};
                const float2 G[R + 1] = {ld2(C, F_G, -1), ld2(C, F_G), ld2(C, F_G, 1)};
                if (hor) {
                    const float2 qd[R + 1] = {ld2(Dn, F_Q1, -1), ld2(Dn, F_Q1), ld2(Dn, F_Q1, 1)};
                    const float2 Wd[R + 1] = {ld2(Dn, F_WP, -1), ld2(Dn, F_WP), ld2(Dn, F_WP, 1)};
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        v2[r] = face_y(st, t, j + r, qc[r + 1], qc[r], qu[r + 1], qu[r], qd[r + 1], qd[r], V[r], G[r + 1], G[r],
                                       U[r + 1], U[r], W[r + 1], Wd[r + 1], W[r], Wd[r], fv[r]);
                        u2[r] = face_x(st, t, j + r, qc[r + 1], qc[r + 2], qc[r], qu[r + 1], qd[r + 1], U[r + 1], G[r + 1], V[r],
                                       V[r + 1], W[r + 1], Wd[r + 1]);
                    }
                }
#pragma unroll
                for (int r = 0; r < R; r++) w2[r] = fz[r] = zero2;
                if (ST || t < nz - 1) {
                    const float2 Vu[R + 1] = {ld2(Up, F_V), ld2(Up, F_V, 1), ld2(Up, F_V, 2)};
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        w2[r] = face_z(j + r, n_dz[r], qc[r + 1], qu[r + 1], qc[r + 2], qc[r], qu[r + 2], qu[r], W[r + 1],
                                       G[r + 1], ld2(Up, F_G, r), U[r + 1], ld2(Up, F_U, r), V[r], V[r + 1], Vu[r],
                                       Vu[r + 1]);
                        if constexpr (FCT) fz[r] = lflux<M>(qc[r + 1], qu[r + 1], w2[r], nz2);
                    }
                }
            }
            if (ST || t + 2 <= l1) {
#pragma unroll
                for (int r = 0; r < R; r++) st2(at4(own, t + 2), F_Q1, q1n[r], r);
            }
            if (FCT && hor) {
#pragma unroll
                for (int r = 0; r < R; r++) st2(own, S_FV, fv[r], r);
            }
            if (ST || t - 1 >= ka) st2(own, S_FY, vs);   // for the row south of the first: its north faces
        } else {
            // the halo warp: south faces of row 25 (limited, for row 24's north
            // faces), P0 of its four rows, south faces of rows 2, 25 and 26
            if (ST || t - 1 >= ka) {
                Split v;
                if constexpr (FCT)
                    v = limit<M>(v2[0], ld2(top, S_BYI), ld2(top, S_BYO, -1), ld2(top, S_BYI, -1), ld2(top, S_BYO));
                else v = split<M>(v2[0]);
                st2(top, S_FY, join<M>(v));
            }
            landed = wait_mine(n);
            if (ST || t + 2 <= l1) donor_halo(t + 2);
            if (hor) {
#pragma unroll 1
                for (int q = 0; q < 3; q++) {
                    const int yr = q == 0 ? 2 : YB - 1 + q;
                    float2 f;
                    const float2 v = face_y_row(st, t, yr, f);
                    if (q == 1) v2[0] = v;
                    if constexpr (FCT) st2(sm + yr * PW + X, S_FV, f);
                }
            }
        }
        // every thread is past I1 of t and the batch of iteration n has
        // landed (or the CTA stops): the planes that batch n+1 overwrites (q0
        // of t-4, the others of t-1) are free
        if (__syncthreads_and(landed ? 1 : 0) == 0) return drain(n);
        if (threadIdx.x == 0 && (ST || t < kb)) issue(t + 1);

        // own-column values for the next iteration and this one's store
        if (ST || t + 3 <= l1) {
            const int L = ST ? min(t + 3, l1) : t + 3;   // (the last middle iteration loads a level it has no use for)
            load_ahead(L);
            if (halo) load_ahead_b(L);
        }
        if (halo) {
            if (FCT && hor) {
#pragma unroll 1
                for (int q = 0; q < 2; q++) {
                    const int yr = q == 0 ? 2 : PH - 3;
                    float *at = sm + yr * PW + X;
                    const float *Q1 = at4(at, t), *Q0 = atq(at, t);
                    float2 bi, bo;
                    betas_y(y0 + yr, at, ld2(Q1, F_Q1), ld2(Q0, 0), ld2(Q1, F_Q1, -1), ld2(Q0, 0, -1), ld2(Q1, F_Q1, 1),
                            ld2(Q0, 0, 1), ld2(at, S_FV), bi, bo);
                    st2(at, S_BYI, bi);
                    st2(at, S_BYO, bo);
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (ST || t + 1 <= tl) n_dz[r] = ldcol(p.dz, rowc[r], t + 1);
                if (ST || t - 1 >= ka) djr_m[r] = ldcol(p.DJR, rowc[r], t - 1);
            }
            const float *C = at4(own, t), *Up = at4(own, t + 1), *Dn = at4(own, t - 1);
            float2 pbi[R], pbo[R];   // the z betas of t-1
#pragma unroll
            for (int r = 0; r < R; r++) {
                pbi[r] = bzi[r];
                pbo[r] = bzo[r];
            }
            // ---- P2: limiter betas at level t --------------------------------
            if (FCT && (ST || (t <= tl && t >= ka - 1))) {
                const float *Q0 = atq(own, t);
                const float2 qc[R + 2] = {ld2(C, F_Q1, -1), ld2(C, F_Q1), ld2(C, F_Q1, 1), ld2(C, F_Q1, 2)};
                const float2 q0[R + 2] = {ld2(Q0, 0, -1), ld2(Q0, 0), ld2(Q0, 0, 1), ld2(Q0, 0, 2)};
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float2 q = qc[r + 1], hi = max2(q, q0[r + 1]), lo = min2(q, q0[r + 1]);
                    if (hor) {
                        // x lines: faces ia, ib, ib+1
                        {
                            const float2 fl = lflux<M>(lft(q), q, u2[r], nz2), fr = rgt(fl);
                            float2 hl = lft(hi), hr = rgt(hi), ll = lft(lo), lr = rgt(lo), hc = hi, lc = lo;
                            float2 afl = fl, afr = fr;
                            if (!INT) {
                                // line ends: the first cell's bounds omit the cell before it;
                                // the last cell's omit the cell after it and its own old
                                // value; both have no flux sums
                                if (ia == 0) { hl.x = hi.x; ll.x = lo.x; }
                                if (ib == 0) { hl.y = hi.y; ll.y = lo.y; }
                                if (ia == nx - 1) { hc.x = lc.x = hr.x = lr.x = q.x; }
                                if (ib == nx - 1) { hc.y = lc.y = hr.y = lr.y = q.y; }
                                if (ia == 0 || ia == nx - 1) afl.x = afr.x = 0.0f;
                                if (ib == 0 || ib == nx - 1) afl.y = afr.y = 0.0f;
                            }
                            betas<M>(max2(max2(hl, hc), hr), min2(min2(ll, lc), lr), q, afl, afr, bxi[r], bxo[r]);
                        }
                        // y lines: faces j and j+1
                        betas_y(j + r, own + r * PW, q, q0[r + 1], qc[r], q0[r], qc[r + 2], q0[r + 2],
                                lflux<M>(qc[r], q, v2[r], nz2), byi[r], byo[r]);
                    }
                    // z line of the own column (its ends keep their fluxes)
                    {
                        float2 hd = hi, ld = lo, hu = hi, lu = lo, hc = hi, lc = lo, fr = fz[r];
                        if (ST || t > 0) {
                            const float2 qd = ld2(Dn, F_Q1, r), q0d = ld2(atq(own, t - 1), 0, r);
                            hd = max2(qd, q0d);
                            ld = min2(qd, q0d);
                        }
                        if (ST || t < nz - 1) {
                            const float2 qu = ld2(Up, F_Q1, r), q0u = ld2(atq(own, t + 1), 0, r);
                            hu = max2(qu, q0u);
                            lu = min2(qu, q0u);
                        } else {
                            hc = lc = hu = lu = q;
                            fr = fzb[r];
                        }
                        betas<M>(max2(max2(hd, hc), hu), min2(min2(ld, lc), lu), q, fzb[r], fr, bzi[r], bzo[r]);
                    }
                }
            }
            // ---- level t-1: the limited flux through its top, the update ---------
            if (ST || t >= ka) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    float2 ft = zero2;
                    const float2 qd = ld2(Dn, F_Q1, r);   // q1 of t-1
                    if (ST || (t >= 1 && t < nz)) {
                        const float2 qc = ld2(C, F_Q1, r);
                        if constexpr (FCT) ft = flux<M>(qd, qc, limit<M>(w2b[r], bzi[r], pbo[r], pbi[r], bzo[r]), nz2);
                        else ft = flux<M>(qd, qc, split<M>(w2b[r]), nz2);
                    } else if (M == A_IEEE && t >= 1) {
                        ft = mul2x(qd, zero2);   // the model top: q times a face velocity of zero
                    }
                    if (ST || t - 1 >= ka) {
                        const int L = t - 1, jr = j + r;
                        float2 hd = hx[r];
                        if (r + 1 == R)
                            hd = ad<M>(hd, north_less<M>(qd, ld2(Dn, F_Q1, R), unjoin<M>(ld2(own, S_FY, R)), fs, nz2));
                        const float2 vd = sb<M>(ft, fb[r]);
                        const float2 G = gm[r];
                        float2 val;
                        if constexpr (M == A_IEEE) {
                            val = sub2x(sub2x(qd, div2x(hd, G)), div2x(vd, djr_m[r]));
                        } else if constexpr (M == A_EXACT) {
                            val = add2(qd, nquot(hd, exdiv(G, S48, R48), tie));
                            val = add2(val, nquot(vd, exdiv(djr_m[r], S48, R48), tie));
                        } else {
                            val = sub2(sub2(qd, mul2(hd, half_of(rcp2(G)))), mul2(vd, half_of(rcp2(djr_m[r]))));
                        }
                        const bool oa = sta && jin(jr), ob = stb && jin(jr);
                        if (!INT) {
                            const bool jring = jr == 0 || jr == ny - 1;
                            const float2 q0L = ld2(atq(own, L), 0, r);
                            if (jring || ia == 0 || ia == nx - 1) val.x = q0L.x;
                            if (jring || ib == 0 || ib == nx - 1) val.y = q0L.y;
                        }
                        if constexpr (M == A_EXACT) worst_of(worst, make_float2(oa ? val.x : 0.0f, ob ? val.y : 0.0f));
                        if (oa || ob) {
                            float *dst = outs + (rowc[r] + (uint32_t)L * lstride);
                            if (oa && ob) *reinterpret_cast<float2 *>(dst) = val;
                            else if (oa) dst[0] = val.x;
                            else dst[1] = val.y;
                        }
                    }
                    fb[r] = ft;
                }
            }
        }
        if (FCT && hor && !halo) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                st2(own, S_BYI, byi[r], r);
                st2(own, S_BYO, byo[r], r);
            }
        }
        if (ST || t < kb) __syncthreads();   // y betas complete; level t-1 is done with
        return true;
    };
#pragma unroll 1
    for (int t = t0; t <= kb; t++) {
        const bool mid = M != A_IEEE && t > ka && t <= l1 - 2 && t < kb;
        if (mid ? !level(std::bool_constant<M != A_IEEE>{}, t) : !level(std::false_type{}, t)) return false;
    }
    return true;
}

// Barrier set-up (threads of the CTA are synchronised by it).
__device__ __forceinline__ void onepass_init_bars(uint64_t *bars)
{
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
}

// Whether a tile's whole plane (origin x0, first output row j0) lies inside
// the domain interior.
__device__ __forceinline__ bool onepass_interior(const Geo &g, int x0, int j0)
{
    return x0 >= 1 && x0 + op::PW - 1 <= g.nx - 2 && j0 - 3 >= 1 && j0 - 3 + op::PH - 1 <= g.ny - 2;
}

// Tile (tx, j0) of a domain, output levels [ka, kb): plane origin and output
// columns, then the march.
template <int M, bool FCT>
__device__ __forceinline__ bool onepass_run(float *sm, uint64_t *bars, const OnePassParams &p, int s, int tx, int j0,
                                            int ka, int kb, bool tie, float &worst)
{
    int x0, xlo, xhi;
    op::xtile(p.g.nx, tx, p.tiles_x, x0, xlo, xhi);
    if (onepass_interior(p.g, x0, j0))
        return onepass_tile<M, FCT, true>(sm, bars, p, s, x0, xlo, xhi, j0, ka, kb, tie, worst);
    return onepass_tile<M, FCT, false>(sm, bars, p, s, x0, xlo, xhi, j0, ka, kb, tie, worst);
}

// The march with IEEE division, out of line, so that it costs the others no
// registers.  A tile of it takes about 2.5 times the exact march's time (up to
// five times with subnormal operands, whose divisions take their slow path).  A
// step of 512x512x40x12 with one wind of 1e-30 takes 3.68 ms where one without
// takes 3.56, with all of v at 1e-30 19.9.  Copies of it for interior tiles
// and for the middle of the march bring that to 19.5 and are left out.
template <bool FCT>
__device__ __noinline__ void onepass_redo(float *sm, uint64_t *bars, const OnePassParams &p, int s, int tx, int j0, int ka,
                                          int kb)
{
    if (threadIdx.x == 0) {
        mbar_inval(&bars[0]);
        mbar_inval(&bars[1]);
    }
    __syncthreads();
    onepass_init_bars(bars);
    float worst = 0.0f;
    int x0, xlo, xhi;
    op::xtile(p.g.nx, tx, p.tiles_x, x0, xlo, xhi);
    onepass_tile<opx::A_IEEE, FCT, false>(sm, bars, p, s, x0, xlo, xhi, j0, ka, kb, false, worst);
}

// Flags of the blocks of columns that the plane with origin (x0, y0) covers, at
// most 3 x 5 of them, one to a lane; every warp asks for itself.  (The votes are
// uniform for the compiler too: answers that were not cost the exact march ten
// spilled registers.)
__device__ __forceinline__ void plane_flags(const OnePassParams &p, int x0, int y0, bool &ieee, bool &tie)
{
    const int nbx = flag_blocks_x(p.g), lane = threadIdx.x & 31;
    const int bx0 = x0 / FLAG_BX, wx = min(x0 + op::PW - 1, p.g.nx - 1) / FLAG_BX - bx0 + 1;
    const int by0 = max(y0, 0) / FLAG_BY, wy = min(y0 + op::PH - 1, p.g.ny - 1) / FLAG_BY - by0 + 1;
    bool b = false, t = false;
    if (lane < wx * wy) {
        const int at = (by0 + lane / wx) * nbx + bx0 + lane % wx, step = p.flags[1];
        b = p.flags[FLAG_HEAD + 2 * at + FLAG_IEEE] == step;
        t = p.flags[FLAG_HEAD + 2 * at + FLAG_TIE] == step;
    }
    ieee = __any_sync(opx::FULL, b);
    tie = __any_sync(opx::FULL, t);
}

// One work item of either form.  A_EXACT: a tile whose fields or values lie
// outside what its quotients are proven for (FLAG_IEEE in its plane, or
// `worst` at the end of the march) is marched with IEEE division; the tile's
// stores are then overwritten, which no other tile reads.
template <int M, bool FCT>
__device__ __forceinline__ void onepass_item(float *sm, uint64_t *bars, const OnePassParams &p, int s, int tx, int j0,
                                             int ka, int kb)
{
    float worst = 0.0f;
    if constexpr (M == opx::A_EXACT) {
        int x0, xlo, xhi;
        op::xtile(p.g.nx, tx, p.tiles_x, x0, xlo, xhi);
        bool redo, tie;
        plane_flags(p, x0, j0 - 3, redo, tie);
        if (!redo) {
            if (!onepass_run<M, FCT>(sm, bars, p, s, tx, j0, ka, kb, tie, worst)) return;
            redo = __syncthreads_or(worst < opx::EXACT_MAX ? 0 : 1) != 0;
        }
        if (redo) onepass_redo<FCT>(sm, bars, p, s, tx, j0, ka, kb);
    } else {
        onepass_run<M, FCT>(sm, bars, p, s, tx, j0, ka, kb, false, worst);
    }
}

// Grid: species fastest, so the CTAs of a tile run together and share its
// wind and metric planes through L2.
template <int M, bool FCT>
__global__ void __launch_bounds__(op::NT, 1) k_mpdata_onepass(const __grid_constant__ OnePassParams p)
{
    using namespace op;
    extern __shared__ float4 smem4[];
    // planes start on 128-byte boundaries (TMA destinations); SMEM has the slack
    float *sm = reinterpret_cast<float *>(smem4) + ((128u - (smem_u32(smem4) & 127u)) & 127u) / sizeof(float);
    __shared__ __align__(8) uint64_t bars[2];
    count_launch(p.flags, blockIdx.x == 0 && threadIdx.x == 0);
    unsigned item;
    int ka, kb;
    split_cta(blockIdx.x, p.whole, p.parts, (unsigned)p.nspecies, p.g.nz, item, ka, kb);
    const int s = (int)(item % (unsigned)p.nspecies), tile = (int)(item / (unsigned)p.nspecies);
    const int tx = tile % p.tiles_x, j0 = (tile / p.tiles_x) * TY;
    __shared__ int stop;
    if (threadIdx.x == 0) stop = *reinterpret_cast<volatile const int *>(p.err);
    __syncthreads();
    if (stop) return;   // an earlier tile of this launch gave up on a TMA wait: stop (the whole CTA)
    onepass_init_bars(bars);
    onepass_item<M, FCT>(sm, bars, p, s, tx, j0, ka, kb);
}

// Batched form: one launch over the work list of (member, species and level
// part, column tile tx, first row j0) items, one CTA per item; params[member]
// holds that member's descriptors, pointers and geometry for the current
// buffer parity.  The hardware block scheduler hands out the items in list
// order as SMs free up.
template <int M, bool FCT>
__global__ void __launch_bounds__(op::NT, 1)
    k_batch_onepass_items(const OnePassParams *__restrict__ params, const int4 *__restrict__ items)
{
    extern __shared__ float4 smem4[];
    float *sm = reinterpret_cast<float *>(smem4) + ((128u - (smem_u32(smem4) & 127u)) & 127u) / sizeof(float);
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ __align__(16) OnePassParams sp;
    __shared__ int stop;
    constexpr int PW4 = (int)(sizeof(OnePassParams) / sizeof(int));
    const int4 w = items[blockIdx.x];
    const int *src = reinterpret_cast<const int *>(params + w.x);
    for (int q = threadIdx.x; q < PW4; q += blockDim.x) reinterpret_cast<int *>(&sp)[q] = src[q];
    // an earlier tile of this launch gave up on a TMA wait: stop (the whole CTA)
    if (threadIdx.x == 0) stop = *reinterpret_cast<volatile const int *>(params[0].err);
    __syncthreads();
    if (stop) return;
    // an item of each member's first species, first level part and first tile
    count_launch(sp.flags, threadIdx.x == 0 && w.y == 0 && w.z == 0 && w.w == 0);
    onepass_init_bars(bars);
    const int k = w.y / op::MAXS;
    const int ka = op::range_begin(sp.g.nz, sp.parts, k), kb = op::range_begin(sp.g.nz, sp.parts, k + 1);
    onepass_item<M, FCT>(sm, bars, sp, w.y % op::MAXS, w.z, w.w, ka, kb);
}

}  // namespace icar
