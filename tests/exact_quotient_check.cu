// Checks, on the device, of the branch-free quotients of the exact kernels
// (opx::nrcp, nquot48, nquot in mpdata_onepass.cuh, std_nrcp and std_quot in
// std_fused.cuh) against the compiler's IEEE division, bit for bit:
//   - the reciprocal for every significand, at exponents over the range of the
//     divisors (metric terms, tracer sums plus 1e-10, flux sums plus 1e-15);
//   - quotients of random operands over the stated ranges, subnormal numerators
//     and quotients among them;
//   - quotients that lie exactly halfway between two subnormal numbers.
// Prints one line per check; exit status 1 on any mismatch.
#include <algorithm>
#include <cstdio>

#include "../hicar_b200/csrc/mpdata_onepass.cuh"
#include "../hicar_b200/csrc/std_fused.cuh"

using namespace icar;
using namespace icar::opx;

enum { RCP, Q48, QUOT, TIE, N_CHECKS };

__device__ unsigned mix(unsigned x)
{
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    return x ^ (x >> 16);
}
// random significand, exponent between lo and hi (down to subnormal), either sign
__device__ float draw(unsigned seed, int lo, int hi)
{
    const unsigned a = mix(seed), b = mix(seed + 0x9e3779b9u);
    const float m = __uint_as_float(0x3f800000u | (a & 0x7fffffu));
    const float v = ldexpf(m, lo + (int)(b % (unsigned)(hi - lo + 1)));
    return (b >> 31) ? -v : v;
}
__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }

__global__ void check(unsigned long long *bad)
{
    const StdArith with_tie{true};
    const unsigned n = gridDim.x * blockDim.x;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < 1u << 23; t += n) {
        // every significand
        for (int e : {-50, -33, -20, -1, 0, 20, 41, 60}) {
            const float b = ldexpf(__uint_as_float(0x3f800000u | t), e);
            const float2 r = nrcp(splat2(b));
            const float want = -(1.0f / b);
            if (differ(r.x, want) || differ(r.y, want) || (e >= -20 && e <= 20 && differ(std_nrcp<true>(b), want)))
                atomicAdd(&bad[RCP], 1ull);
        }
        for (int m = 0; m < 16; m++) {
            // numerators down to the smallest subnormals, divisors of tracer and flux sums; the quotient normal
            const unsigned seed = mix(t * 16u + m);
            float a = draw(seed, -149, 40), b = fabsf(draw(seed + 1u, -50, 41));
            float A = a * 0x1p48f, want = -(A / b);
            if (fabsf(want) >= 0x1p-126f && fabsf(want) < 0x1p120f) {
                const float2 q = nquot48(splat2(a), splat2(b));
                if (differ(q.x, want) || differ(q.y, want)) atomicAdd(&bad[Q48], 1ull);
            }
            // quotients by metric terms, subnormal ones among them
            b = fabsf(draw(seed + 2u, -20, 19));
            a = draw(seed + 3u, m % 2 ? -149 : -40, m % 2 ? -100 : 78);
            const bool tie = tie_divisor(b);
            const ExDiv d = exdiv(splat2(b), S48, R48);
            float2 q = nquot(splat2(a), d, tie);
            const float nr = std_nrcp<true>(b);
            if (differ(q.x, -(a / b)) || differ(q.y, -(a / b)) || differ(std_quot<true>(a, b, nr, {tie}), a / b))
                atomicAdd(&bad[QUOT], 1ull);
            // halfway: b even and not a power of two, a = b (2k+1) 2^-150
            const unsigned half = 3u + mix(seed + 4u) % (m % 4 ? 500u : 500000u);
            b = 2.0f * (float)half;
            const unsigned k = mix(seed + 5u) % ((1u << 24) / half / 2u);
            const unsigned steps = half * (2u * k + 1u);
            if (tie_divisor(b) && steps < 1u << 24) {
                a = (seed & 1u) ? -__uint_as_float(steps) : __uint_as_float(steps);
                const ExDiv e = exdiv(splat2(b), S48, R48);
                q = nquot(splat2(a), e, true);
                if (differ(q.x, -(a / b)) || differ(q.y, -(a / b)) ||
                    differ(std_quot<true>(a, b, std_nrcp<true>(b), with_tie), a / b))
                    atomicAdd(&bad[TIE], 1ull);
            }
        }
    }
}

int main()
{
    unsigned long long *d = nullptr, bad[N_CHECKS] = {};
    if (cudaMalloc(&d, sizeof(bad)) != cudaSuccess || cudaMemset(d, 0, sizeof(bad)) != cudaSuccess) return 2;
    check<<<148 * 8, 256>>>(d);
    if (cudaMemcpy(bad, d, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    const char *name[N_CHECKS] = {"reciprocal", "scaled quotient", "quotient", "halfway"};
    bool any = false;
    for (int c = 0; c < N_CHECKS; c++) {
        std::printf("%s mismatches=%llu\n", name[c], bad[c]);
        any |= bad[c] != 0;
    }
    return any;
}
