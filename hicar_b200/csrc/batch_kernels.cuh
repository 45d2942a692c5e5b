// Batched form: many independent domains (ensemble members or served
// requests) of uneven nx x ny x nz advance together.  One step is three
// launches whatever the number of members, captured once in a CUDA graph:
//   k_batch_forcing        relaxation-zone update of every forced species
//   k_batch_prep           species-independent per-step fields of every member
//   k_batch_onepass_items  the single-pass kernel over the (member, species,
//                          tile, level range) work list (mpdata_onepass.cuh)
// Member data lives in a device table (BatchMember); the simple kernels map
// their flat block index to a member by binary search over per-member block
// prefix sums.
#pragma once
#include "boundary_kernels.cuh"
#include "common.cuh"
#include "mpdata_fused.cuh"

namespace icar {

constexpr int BATCH_MAX_SPECIES = 32;

struct BatchMember {
    Geo g;
    float dx, dt;
    double dtd;
    int S, adv_den, nzone;
    int *flags;
    const float *u, *v, *w, *rho, *jac, *ju, *jv, *jw, *dz;
    float *Um, *Vm, *Wm, *Gc, *DJR, *Wp;
    const float *filter;
    const int *zone;
    const float *q0[BATCH_MAX_SPECIES];
    float *out[BATCH_MAX_SPECIES];
    float *forcing[BATCH_MAX_SPECIES];
    const float *dqdt[BATCH_MAX_SPECIES];
};

// index of the last prefix entry <= b (prefix[0] = 0, prefix[n] = total)
__device__ __forceinline__ int find_owner(const int *__restrict__ prefix, int n, int b)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// pairs[p] = (member, species) of the p-th forced species; prefix over their
// blocks of ceil(nzone*nz/256).
__global__ void k_batch_forcing(const BatchMember *__restrict__ mem, const int *__restrict__ prefix,
                                const int2 *__restrict__ pairs, int npairs)
{
    const int p = find_owner(prefix, npairs, blockIdx.x);
    const int2 ms = pairs[p];
    const BatchMember &m = mem[ms.x];
    const size_t t = (size_t)(blockIdx.x - prefix[p]) * blockDim.x + threadIdx.x;
    const Geo g = m.g;
    if (t >= (size_t)m.nzone * g.nz) return;
    const int z = (int)(t % (size_t)m.nzone);
    const int k = (int)(t / (size_t)m.nzone);
    const int packed = m.zone[z];
    const int i = packed % g.nx, j = packed / g.nx;
    const size_t c = ix(g, i, k, j);
    float *q = const_cast<float *>(m.q0[ms.y]);
    float *fo = m.forcing[ms.y];
    const float fnew = (float)((double)fo[c] + (double)m.dqdt[ms.y][c] * m.dtd);
    fo[c] = fnew;
    const float flt = m.filter[packed];
    if (flt == 1.0f)
        q[c] = fnew;
    else if (flt < 1.0f)
        q[c] = (float)((double)q[c] + ((double)flt * m.dtd / 3600.0) * (double)(fnew - q[c]));
}

// prefix over members of ceil(prep_quads/256) blocks
__global__ void __launch_bounds__(256)
    k_batch_prep(const BatchMember *__restrict__ mem, const int *__restrict__ prefix, int nmem)
{
    const int mi = find_owner(prefix, nmem, blockIdx.x);
    const BatchMember &m = mem[mi];
    const PrepFields f{m.u, m.v, m.w, m.rho, m.jac, m.ju, m.jv, m.jw, m.dz, m.Um, m.Vm, m.Wm, m.Gc, m.DJR, m.Wp};
    prep_quad(m.g, m.dx, m.dt, m.adv_den, f, (blockIdx.x - prefix[mi]) * blockDim.x + threadIdx.x, m.flags);
}

}  // namespace icar
