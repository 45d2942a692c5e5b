// How a launch of the single-pass MPDATA kernel divides its column tiles among
// the SMs (one CTA each at a time): the first `whole` tiles march whole columns,
// the others are cut into `parts` ranges of levels, equal to one level, each a
// CTA of its own.  Host arithmetic only; CTAs are handed out in order, the whole
// columns first.
//
// A CTA that marches only part of a column repeats about three levels of its
// neighbours' work, and its start-up costs about two more.  So a cut pays only
// where whole columns would leave SMs idle, which is in the last wave: either
// everything is cut (short launches), or what is left after the full waves, or
// that and one full wave more, whichever makes the launch shortest by
// waves x (levels + overhead); ranges have at least MIN_RANGE levels.  With the
// cut of all columns or none, as it was before, a launch a little above a whole
// number of waves cost one wave more.  Whole steps in fast arithmetic: 96x250x35
// with 7 species (168 tiles) 222 -> 179 us, 512x400x40 with one (171) 329 -> 293,
// 256x256x40 with 5 (300) 397 -> 336, 250x210x40 with 12 (600) 686 -> 598, 128x128x20
// with one (18, all cut) 40, 187x301x33 with 5 (280, nothing cut) 278.
#pragma once

namespace icar {
namespace op {

constexpr int MIN_RANGE = 5;

struct ColumnSplit {
    long whole;
    int parts;
};

#ifdef __CUDACC__
__host__ __device__
#endif
inline int range_begin(int nz, int parts, int k) { return (int)((unsigned)nz * (unsigned)k / (unsigned)parts); }

// cost of marching `tiles` tiles of nz levels in `parts` ranges each, in levels
inline long march_cost(long tiles, int nz, int parts, int sms)
{
    return (tiles * parts + sms - 1) / sms * ((nz + parts - 1) / parts + 2 + (parts > 1 ? 3 : 0));
}

inline int best_parts(long tiles, int nz, int sms)
{
    int best = 1;
    for (int n = 2; nz / n >= MIN_RANGE; n++)
        if (march_cost(tiles, nz, n, sms) < march_cost(tiles, nz, best, sms)) best = n;
    return best;
}

inline ColumnSplit split_columns(long tiles, int nz, int sms)
{
    ColumnSplit best{0, best_parts(tiles, nz, sms)};
    long least = march_cost(tiles, nz, best.parts, sms);
    for (long whole = tiles / sms * sms, n = 0; whole > 0 && n < 2; whole -= sms, n++) {
        const int parts = best_parts(tiles - whole, nz, sms);
        const long cost = march_cost(whole, nz, 1, sms) + march_cost(tiles - whole, nz, parts, sms);
        if (cost < least) {
            least = cost;
            best = {whole, parts};
        }
    }
    return best;
}

// CTAs of the launch, and the tile and level range [ka, kb) of CTA b
inline long split_ctas(const ColumnSplit &s, long tiles) { return s.whole + (tiles - s.whole) * s.parts; }
#ifdef __CUDACC__
__host__ __device__
#endif
inline void split_cta(unsigned b, unsigned whole, int parts, unsigned tiles, int nz, unsigned &tile, int &ka, int &kb)
{
    if (b < whole) {
        tile = b, ka = 0, kb = nz;
    } else {
        const unsigned cut = tiles - whole, k = (b - whole) / cut;   // all first ranges, then all second ones, ...
        tile = whole + (b - whole) % cut;
        ka = range_begin(nz, parts, (int)k);
        kb = range_begin(nz, parts, (int)k + 1);
    }
}

}  // namespace op
}  // namespace icar
