// Wind balance and the stable time step on the device: the two per-step
// wind operations that sit next to advection in ICAR's time loop.
//
//   k_balance_uvw   balance_uvw (src/physics/wind.f90:88-164) with
//                   calc_divergence(horz_only) and calc_w (:166-271): one
//                   thread per column marches up it, forming the
//                   horizontal divergence of the metric-weighted u, v at
//                   each level and integrating w from w = 0 below the ground;
//                   the levels arrive in shared-memory planes ahead of use.
//   k_dt_maxima     the maxima compute_dt (src/main/time_step.f90:51-168)
//                   needs: max |u|, |v|, |w| over the whole arrays and the
//                   per-cell CFL rate max(|u|/dx, |v|/dx, |w|/dz) over the
//                   tile, reduced in the block and combined with atomicMax
//                   on the bit patterns (order-preserving for values >= 0).
//
// Both are single passes over the fields (HBM bound); the expressions keep
// the Fortran evaluation order, like the advection kernels.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "common.cuh"
#include "mpdata_fused.cuh"

namespace icar {

namespace balf {
// CTA tile: 32 x 8 columns, one thread per column marching up k.  The seven fields a level needs (u, J_u, v, J_v, rho, dz, J_w) arrive
// in shared-memory planes by 16-byte cp.async, DEPTH levels ahead of use:
// each plane spans x from i0-4 (a multiple of 4) to i0+35 and y from j0-1
// to j0+8, covering the faces i0..i0+32 / j0..j0+8 and the density
// neighbours the face weights read.
constexpr int BX = 32, BY = 8, NT = BX * BY;
constexpr int PW = 40, PH = BY + 2, PLANE = PW * PH;
constexpr int NF = 7;                      // u, ju, v, jv, rho, dz, jw
constexpr int DEPTH = 3, NSLOT = DEPTH + 1;
constexpr int CPR = PW / 4, NCH = (NF * CPR * PH + NT - 1) / NT;
constexpr size_t SMEM = (size_t)NSLOT * NF * PLANE * sizeof(float);
}  // namespace balf

// Columns i_s..i_e x j_s..j_e (its-1..ite+1 clipped to the domain, i.e.
// [max(hs-1,0), min(n-hs,n-1)] for one image with halo hs) get the balanced
// w; every other column gets w = 0 (calc_w sets the whole array first).
//
// Face values: u*J_u times the face density when ADV (the outermost faces
// extrapolate it), wind.f90:237-239; v*J_v likewise, :241-243.  EDGE tiles
// touch the domain's sides, the others have no outermost face.
//
// 334 MB at 512x512x40 (51 us at the measured copy rate), bound by issue there
// and by the latency of the march on domains of up to a wave of tiles.  The
// density is a template argument and tiles inside the domain carry no side
// conditions: 80 us with density and 73 without at 512x512x40, 33 both at
// 25x38x54, where a run-time switch and side conditions everywhere took 97 and
// 75, 47 and 37.  Two columns per thread share operands but march slower: 84
// and 84, 42 and 45.
template <bool ADV, bool EDGE>
__device__ __forceinline__ void balance_march(float *sm, const Geo &g, int hs, float dx, int i0, int j0,
                                              const float *__restrict__ u, const float *__restrict__ v,
                                              const float *__restrict__ rho, const float *__restrict__ dz,
                                              const float *__restrict__ ju, const float *__restrict__ jv,
                                              const float *__restrict__ jw, float *__restrict__ w)
{
    using namespace balf;
    const int tx = threadIdx.x % BX, ty = threadIdx.x / BX;
    const int i = i0 + tx, j = j0 + ty;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int ox = i0 - 4, oy = j0 - 1;
    const int i_s = max(hs - 1, 0), i_e = min(nx - hs, nx - 1);
    const int j_s = max(hs - 1, 0), j_e = min(ny - hs, ny - 1);
    // every thread's chunks of one level: field f, row ly, chunk cx
    const float *src[NCH];
    int dst[NCH];
    unsigned okm = 0u;
#pragma unroll
    for (int c = 0; c < NCH; c++) {
        const int e = threadIdx.x + c * NT;
        dst[c] = -1;
        src[c] = u;
        if (e < NF * CPR * PH) {
            const int f = e / (CPR * PH), r = e % (CPR * PH);
            const int ly = r / CPR, cx = r % CPR;
            const int gi = ox + 4 * cx, gj = oy + ly;
            const bool yface = f == 2 || f == 3;
            dst[c] = f * PLANE + ly * PW + 4 * cx;
            const float *base = f == 0 ? u : f == 1 ? ju : f == 2 ? v : f == 3 ? jv : f == 4 ? rho : f == 5 ? dz : jw;
            if (gi >= 0 && gi < g.P && gj >= 0 && gj < (yface ? ny + 1 : ny)) {
                okm |= 1u << c;
                src[c] = base + (size_t)gi + (size_t)g.P * nz * gj;
            }
        }
    }
    auto issue = [&](int k) {
        if (k < nz) {
            float *slot = sm + (size_t)(k % NSLOT) * NF * PLANE;
#pragma unroll
            for (int c = 0; c < NCH; c++)
                if (dst[c] >= 0) {
                    const bool ok = (okm >> c) & 1u;
                    cp_async16(slot + dst[c], src[c], ok);
                    if (ok) src[c] += g.P;
                }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int k = 0; k < DEPTH; k++) issue(k);
    const bool in = i < nx && j < ny;
    const bool bal = in && i >= i_s && i <= i_e && j >= j_s && j <= j_e;
    float wb = 0.0f, rib = 0.0f, jwb = 0.0f;  // w, interface density and J_w one level down
    float *wp = w + (in ? ix(g, i, 0, j) : 0);
    const int pc = (ty + 1) * PW + tx + 4;
    for (int k = 0; k < nz; k++) {
        cp_async_wait<DEPTH - 2>();  // levels k and k+1 have landed
        __syncthreads();
        issue(k + DEPTH);            // into the slot of level k-1, read by nobody any more
        // Outside the domain the metrics are zeros, and a quotient of zeros
        // takes the division's slow path: those columns are skipped.
        if (EDGE && !bal) {
            if (in) *wp = 0.0f;
            wp += g.P;
            continue;
        }
        const float *L = sm + (size_t)(k % NSLOT) * NF * PLANE + pc;
        const float *Lu = sm + (size_t)((k + 1) % NSLOT) * NF * PLANE + pc;
        const float *U = L, *JU = L + PLANE, *V = L + 2 * PLANE, *JV = L + 3 * PLANE, *R = L + 4 * PLANE;
        float rs = 0.0f, rc = 0.0f, rn = 0.0f;  // density here and in the rows beside
        if (ADV) {
            rs = R[-PW];
            rc = R[0];
            rn = R[PW];
        }
        const float sj = V[0] * JV[0], nj = V[PW] * JV[PW];
        float vs = sj, vn = nj;
        if (ADV) {
            vs = sj * (rs + rc) / 2.0f;
            if (EDGE && j == 0) vs = sj * (1.5f * rc - 0.5f * rn);
            vn = nj * (rc + rn) / 2.0f;
            if (EDGE && j + 1 == ny) vn = nj * (1.5f * rc - 0.5f * rs);
        }
        const float ej = U[1] * JU[1], wj = U[0] * JU[0];
        float ue = ej, uw = wj;
        if (ADV) {
            const float rl = R[-1], rr = R[1];
            ue = ej * (rc + rr) / 2.0f;
            uw = wj * (rl + rc) / 2.0f;
            if (EDGE && i + 1 == nx) ue = ej * (1.5f * rc - 0.5f * rl);
            if (EDGE && i == 0) uw = wj * (1.5f * rc - 0.5f * rr);
        }
        const float div = ((ue - uw) + (vn - vs)) / dx;
        const float d = L[5 * PLANE], jwc = L[6 * PLANE];
        float wk;
        if (ADV) {
            // rho_i(k) = (rho_k*dz_k + rho_k+1*dz_k+1) / (dz_k + dz_k+1), wind.f90:175-176
            float ri = rc;
            if (k < nz - 1) {
                const float dzu = Lu[5 * PLANE];
                ri = (rc * d + Lu[4 * PLANE] * dzu) / (d + dzu);
            }
            wk = ((k == 0 ? 0.0f : wb * rib * jwb) - div * d) / (jwc * ri);
            rib = ri;
        } else {
            wk = ((k == 0 ? 0.0f : wb * jwb) - div * d) / jwc;
        }
        wb = wk;
        jwb = jwc;
        if (in) *wp = bal ? wk : 0.0f;
        wp += g.P;
    }
    cp_async_wait<0>();
}

template <bool ADV>
__global__ void __launch_bounds__(balf::NT)
    k_balance_uvw(Geo g, int hs, float dx, const float *__restrict__ u, const float *__restrict__ v,
                  const float *__restrict__ rho, const float *__restrict__ dz, const float *__restrict__ ju,
                  const float *__restrict__ jv, const float *__restrict__ jw, float *__restrict__ w)
{
    extern __shared__ float4 sm4[];
    float *sm = reinterpret_cast<float *>(sm4);
    const int i0 = blockIdx.x * balf::BX, j0 = blockIdx.y * balf::BY;
    if (i0 > 0 && j0 > 0 && i0 + balf::BX < g.nx && j0 + balf::BY < g.ny)
        balance_march<ADV, false>(sm, g, hs, dx, i0, j0, u, v, rho, dz, ju, jv, jw, w);
    else
        balance_march<ADV, true>(sm, g, hs, dx, i0, j0, u, v, rho, dz, ju, jv, jw, w);
}

// out[0..2] = bits of max |u|, |v|, |w| over the arrays plus one; out[3] =
// bits of the largest per-cell rate over the tile (i, j in [hs, n-1-hs], every
// k).  out must be zero on entry.  dzl is dz_levels (nz).
//
// A NaN among other values is skipped; of an array that holds nothing else
// out stays zero, which dt_from_maxima turns into a NaN again.  So every
// maximum starts as NaN ("nothing yet") and grows by fmaxf, which returns the
// other operand for a NaN.
//
// Bound by reading the three fields.  Rounded division by a positive number
// is monotone, so the largest rate is the largest speed divided: of u over
// the tile's x faces [hs, nx-hs] and of v over its y faces by dx, once per
// block, and of w over a row of level k by the thickness of level k and (its
// top face being the bottom face of the next cell) of level k+1, once per
// thread and row.  So no value is read twice or divided by itself, and a warp
// reads its row of u, v and w in 16-byte pieces.  With one value per thread,
// three divisions each and indices from 64-bit divisions the call took 176 us
// at 512x512x40; it takes 57 now, of which reading 126 MB has to take 19 and
// the small copies and the wait for the result are most of the rest.
namespace dtm {
constexpr int NT = 256, WARPS = NT / 32, U = 2;
}

// mx: maximum so far over the whole row; tx: over x in [a, b] (b < n); both over x < n
__device__ __forceinline__ void dt_take(float4 v, int i, int n, int a, int b, bool tile, float &mx, float &tx)
{
    const float f[4] = {fabsf(v.x), fabsf(v.y), fabsf(v.z), fabsf(v.w)};
#pragma unroll
    for (int m = 0; m < 4; m++) {
        if (i + m < n) mx = fmaxf(mx, f[m]);
        if (tile && i + m >= a && i + m <= b) tx = fmaxf(tx, f[m]);
    }
}

__global__ void __launch_bounds__(dtm::NT)
    k_dt_maxima(Geo g, int hs, float dx, const float *__restrict__ u, const float *__restrict__ v,
                const float *__restrict__ w, const float *__restrict__ dzl, unsigned *__restrict__ out)
{
    using namespace dtm;
    __shared__ float part[4][WARPS];
    const int nx = g.nx, ny = g.ny, nz = g.nz, nq = g.P / 4;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const unsigned row = blockIdx.x * WARPS + warp;  // k + nz*j, j <= ny (v has ny+1 rows)
    const int j = (int)(row / (unsigned)nz), k = (int)(row - (unsigned)j * nz);
    const float none = __int_as_float(0x7fffffff);
    float mu = none, mv = none, mw = none, tu = none, tv = none, tw = none;
    if (j <= ny) {
        const bool cells = j < ny, tile = j >= hs && j <= ny - 1 - hs, vtile = j >= hs && j <= ny - hs;
        const float4 *pu = reinterpret_cast<const float4 *>(u + (size_t)row * g.P);
        const float4 *pv = reinterpret_cast<const float4 *>(v + (size_t)row * g.P);
        const float4 *pw = reinterpret_cast<const float4 *>(w + (size_t)row * g.P);
        const float4 blank = make_float4(none, none, none, none);
        for (int q0 = lane; q0 < nq; q0 += 32 * U) {
            float4 a[U], b[U], c[U];
#pragma unroll
            for (int m = 0; m < U; m++) {
                const int q = q0 + 32 * m;
                const bool in = q < nq;
                a[m] = in && cells ? pu[q] : blank;
                b[m] = in ? pv[q] : blank;
                c[m] = in && cells ? pw[q] : blank;
            }
#pragma unroll
            for (int m = 0; m < U; m++) {
                const int i = 4 * (q0 + 32 * m);
                dt_take(a[m], i, nx + 1, hs, nx - hs, tile && hs <= nx - 1 - hs, mu, tu);
                dt_take(b[m], i, nx, hs, nx - 1 - hs, vtile && hs <= ny - 1 - hs, mv, tv);
                dt_take(c[m], i, nx, hs, nx - 1 - hs, tile, mw, tw);
            }
        }
    }
    float m3 = 0.0f;
    if (tw > 0.0f) {
        m3 = fmaxf(tw / dzl[k], m3);
        if (k + 1 < nz) m3 = fmaxf(tw / dzl[k + 1], m3);
    }
    m3 = fmaxf(fmaxf(tu, tv) / dx, m3);
    for (int o = 16; o > 0; o >>= 1) {
        mu = fmaxf(mu, __shfl_xor_sync(0xffffffffu, mu, o));
        mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
        mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, o));
        m3 = fmaxf(m3, __shfl_xor_sync(0xffffffffu, m3, o));
    }
    if (lane == 0) {
        part[0][warp] = mu;
        part[1][warp] = mv;
        part[2][warp] = mw;
        part[3][warp] = m3;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        float m = none;
        for (int o = 0; o < WARPS; o++) m = fmaxf(m, part[threadIdx.x][o]);
        // the values there only grow: no atomic where it could not change them
        const unsigned bits = threadIdx.x == 3 ? __float_as_uint(m) : m >= 0.0f ? __float_as_uint(m) + 1u : 0u;
        if (bits > *reinterpret_cast<volatile unsigned *>(&out[threadIdx.x])) atomicMax(&out[threadIdx.x], bits);
    }
}

// The maxima from k_dt_maxima's words: max |u|, |v|, |w| (NaN for an array of
// NaN) and the largest rate, NaN where one of the winds is.
inline void decode_maxima(const unsigned bits[4], float m[4])
{
    for (int i = 0; i < 4; i++) {
        const unsigned b = i < 3 && bits[i] ? bits[i] - 1u : bits[i];
        memcpy(&m[i], &b, sizeof(b));
        if (i < 3 && !bits[i]) m[i] = NAN;
    }
    if (m[0] != m[0] || m[1] != m[1] || m[2] != m[2]) m[3] = NAN;
}

// compute_dt's combination of the maxima for cfl_strictness 1..5 (host
// side, same FP32 operations as the reference; a NaN stays one).  use_density:
// the reference's density-weighted terms are commented out, so the winds then
// contribute nothing and dt is infinite.
inline float dt_from_maxima(const float m[4], float cfl, int strictness, int use_density)
{
    const float three_d_cfl = 0.577350269f;
    const float sqrt3 = std::sqrt(3.0f) * 1.001f;
    float maxwind1d = 0.0f, maxwind3d = 0.0f;
    auto mx = [](float a, float b) { return a > b || a != a ? a : b; };
    if (strictness == 1) {
        if (!use_density) maxwind1d = mx(mx(m[0], m[1]), m[2]);
        maxwind3d = maxwind1d * sqrt3;
    } else if (strictness == 5) {
        if (!use_density) maxwind3d = m[0] + m[1] + m[2];
    } else {
        if (!use_density) maxwind3d = m[3];
        if (strictness == 2) {
            maxwind3d = maxwind3d * three_d_cfl;
            if (!use_density) maxwind1d = mx(mx(m[0], m[1]), m[2]);
            maxwind3d = mx(maxwind1d, maxwind3d);
        } else if (strictness == 4) {
            maxwind3d = maxwind3d * sqrt3;
        }
    }
    return cfl / maxwind3d;
}

}  // namespace icar
