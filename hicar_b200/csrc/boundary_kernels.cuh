// Lateral-boundary update and clipping for the advected species.
//   k_apply_forcing   apply_forcing, advected 3-D branch, src/objects/domain_obj.f90:3495-3506
//   k_enforce_limits  enforce_limits, src/objects/domain_obj.f90:3124-3147
#pragma once
#include "common.cuh"

namespace icar {

// Relaxation-zone update over the columns whose filter is non-zero (zone[]
// holds their (i,j) packed as i + nx*j), for every species that has forcing
// in one launch.  dt is
// the real64 dt%seconds(); the Fortran expression mixes real and real64, so
// it is evaluated in double and rounded on assignment.  Columns with filter
// 0 are left alone: the reference adds 0*(forcing-q) there, which leaves q
// unchanged for finite inputs.  Forcing values are advanced only inside the
// zone, the only place the advected species read them.
struct ForcingPtrs {
    float *q[32];
    float *forcing[32];
    const float *dqdt[32];
};

// Bound by the zone's sectors (five accesses a value, rows as short as nine
// values at the east and west sides).  A thread takes FORCE_LEVELS levels of
// one zone column, so the column's place and weight are formed once for them
// and their loads are in flight together; blockIdx.y is the level group and
// blockIdx.z the species.  One level per thread with three 64-bit divisions
// took 64 us for 12 species of 512x512x40, this takes 45.
constexpr int FORCE_LEVELS = 4;

__global__ void __launch_bounds__(256)
    k_apply_forcing(Geo g, int nzone, const int *__restrict__ zone, const float *__restrict__ filter2d, double dt,
                    const __grid_constant__ ForcingPtrs fp)
{
    const int z = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (z >= nzone) return;
    float *q = fp.q[blockIdx.z], *forcing = fp.forcing[blockIdx.z];
    const float *dqdt = fp.dqdt[blockIdx.z];
    const int packed = zone[z];
    const int i = packed % g.nx, j = packed / g.nx, k0 = (int)blockIdx.y * FORCE_LEVELS;
    const size_t c = ix(g, i, k0, j);
    const float flt = filter2d[packed];
    float f[FORCE_LEVELS], d[FORCE_LEVELS], o[FORCE_LEVELS];
#pragma unroll
    for (int m = 0; m < FORCE_LEVELS; m++) {
        f[m] = d[m] = o[m] = 0.0f;
        if (k0 + m < g.nz) {
            f[m] = forcing[c + (size_t)m * g.P];
            d[m] = dqdt[c + (size_t)m * g.P];
            if (flt < 1.0f) o[m] = q[c + (size_t)m * g.P];
        }
    }
    const double weight = (double)flt * dt / 3600.0;
#pragma unroll
    for (int m = 0; m < FORCE_LEVELS; m++)
        if (k0 + m < g.nz) {
            const float fnew = (float)((double)f[m] + (double)d[m] * dt);
            forcing[c + (size_t)m * g.P] = fnew;
            if (flt == 1.0f)
                q[c + (size_t)m * g.P] = fnew;
            else if (flt < 1.0f)
                q[c + (size_t)m * g.P] = (float)((double)o[m] + weight * (double)(fnew - o[m]));
        }
}

// q = max(q, 0) for every species in one launch (blockIdx.y = species), the
// pad columns left alone.  Bound by reading the fields: most values are not
// negative, so a 16-byte group is only stored when one in it is, and only
// then is its position in the row formed.  Four loads in flight per thread;
// one value per thread with its row index formed by a 64-bit division took
// 394 us for 12 species of 512x512x40, this takes 77 (floor of 506 MB read: 77).
struct FieldPtrs {
    float *q[32];
};

namespace lim {
constexpr int NT = 256, U = 4;
}

__global__ void __launch_bounds__(lim::NT) k_enforce_limits(Geo g, size_t quads, FieldPtrs fp)
{
    float4 *q = reinterpret_cast<float4 *>(fp.q[blockIdx.y]);
    const size_t t0 = (size_t)blockIdx.x * (lim::NT * lim::U) + threadIdx.x;
    float4 v[lim::U];
#pragma unroll
    for (int m = 0; m < lim::U; m++)
        if (t0 + m * lim::NT < quads) v[m] = q[t0 + m * lim::NT];
#pragma unroll
    for (int m = 0; m < lim::U; m++) {
        const size_t t = t0 + m * lim::NT;
        if (t >= quads || !(v[m].x < 0.0f || v[m].y < 0.0f || v[m].z < 0.0f || v[m].w < 0.0f)) continue;
        const int i = 4 * (int)(t % (size_t)(g.P / 4));
        float *o = reinterpret_cast<float *>(q + t);
        if (v[m].x < 0.0f && i < g.nx) o[0] = 0.0f;
        if (v[m].y < 0.0f && i + 1 < g.nx) o[1] = 0.0f;
        if (v[m].z < 0.0f && i + 2 < g.nx) o[2] = 0.0f;
        if (v[m].w < 0.0f && i + 3 < g.nx) o[3] = 0.0f;
    }
}

// n (<= 32) fields of one geometry
inline void enforce_limits(const Geo &g, float *const *q, int n, cudaStream_t st)
{
    const size_t quads = (size_t)g.P * g.nz * g.ny / 4, per = lim::NT * lim::U;
    FieldPtrs fp{};
    for (int s = 0; s < n; s++) fp.q[s] = q[s];
    k_enforce_limits<<<dim3((unsigned)((quads + per - 1) / per), (unsigned)n), lim::NT, 0, st>>>(g, quads, fp);
}

}  // namespace icar
