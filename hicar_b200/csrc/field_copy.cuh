// Copies between a caller's contiguous field (x fastest, rows of ex values)
// and the handle's pitched rows, in either direction.
//
// Pure traffic: one read and one write per value.  A 2-D copy of rows that
// short runs at 1.85 TB/s on the copy path, whatever the direction; here a
// block takes whole rows worth 16 KB, every thread has its four 16-byte loads
// in flight before the first store, and 12 species of 512x512x40 move in
// 203 us instead of 546 (floor of 1.01 GB at the measured copy rate: 154).
// Rows that do not start on 16-byte boundaries (ex not a multiple of 4, or an
// unaligned caller's pointer) go value by value, eight in flight, coalesced
// on both sides.
#pragma once
#include <algorithm>

#include "common.cuh"

namespace icar {

namespace rp {
constexpr int NT = 256;
template <class T> constexpr int U = sizeof(T) == 16 ? 4 : 8;  // values of T in flight per thread
// A block's rows: worth NT * U values where that gives every SM two blocks,
// fewer on smaller fields, down to a value per thread: a copy of 35x25x37 took
// 4.1 us among others in 16 blocks with eight values per thread and takes 3.8 (a
// 2-D copy 3.7 to 4.2), 128x128x20 in 80 blocks 4.0 and 3.8 (4.1).
constexpr size_t BLOCKS = 2 * 148;
template <class T> inline size_t rows_per_block(size_t n, size_t rows)
{
    const size_t values = std::min<size_t>(std::max<size_t>(n * rows / BLOCKS, NT), NT * U<T>);
    return std::max<size_t>(1, values / n);
}
}  // namespace rp

// rows x n values of T from src (row stride ss) to dst (row stride ds); a
// block's share is `per` rows.
template <class T>
__global__ void __launch_bounds__(rp::NT) k_repack(const T *src, size_t ss, T *dst, size_t ds, unsigned n, size_t rows,
                                                   unsigned per)
{
    constexpr int U = rp::U<T>;
    const size_t r0 = (size_t)blockIdx.x * per;
    const unsigned total = (unsigned)(rows - r0 < per ? rows - r0 : per) * n;
    src += r0 * ss;
    dst += r0 * ds;
    for (unsigned t0 = threadIdx.x; t0 < total; t0 += rp::NT * U) {
        T v[U];
        size_t to[U];
#pragma unroll
        for (int m = 0; m < U; m++) {
            const unsigned t = t0 + m * rp::NT;
            if (t < total) {
                const unsigned r = t / n, i = t - r * n;
                to[m] = r * ds + i;
                v[m] = src[r * ss + i];
            }
        }
#pragma unroll
        for (int m = 0; m < U; m++)
            if (t0 + m * rp::NT < total) dst[to[m]] = v[m];
    }
}

// Both pointers are this device's memory, 4-byte aligned; strides and ex in
// floats.
inline void repack(const float *src, size_t ss, float *dst, size_t ds, size_t ex, size_t rows, cudaStream_t st)
{
    if (ex == 0 || rows == 0) return;
    if (((uintptr_t)src | (uintptr_t)dst) % 16 == 0 && (ss | ds | ex) % 4 == 0) {
        const size_t per = rp::rows_per_block<float4>(ex / 4, rows);
        k_repack<float4><<<(unsigned)((rows + per - 1) / per), rp::NT, 0, st>>>(
            reinterpret_cast<const float4 *>(src), ss / 4, reinterpret_cast<float4 *>(dst), ds / 4,
            (unsigned)(ex / 4), rows, (unsigned)per);
    } else {
        const size_t per = rp::rows_per_block<float>(ex, rows);
        k_repack<float><<<(unsigned)((rows + per - 1) / per), rp::NT, 0, st>>>(src, ss, dst, ds, (unsigned)ex, rows,
                                                                              (unsigned)per);
    }
}

}  // namespace icar
