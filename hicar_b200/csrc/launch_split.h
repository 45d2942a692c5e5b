// How a launch of the single-pass MPDATA kernel divides its column tiles among
// the SMs (one CTA each at a time): the first `whole` tiles march whole columns,
// the others are cut into `parts` ranges of levels, each a CTA of its own.  Host
// arithmetic only; CTAs are handed out in order, the whole columns first.
//
// A CTA that marches only part of a column repeats about three levels of its
// neighbours' work, and its start-up costs about two more.  So a cut pays only
// where whole columns would leave SMs idle.  A launch short of a wave (or a few
// waves of short columns) is cut as a whole, for the least waves x (levels +
// overhead), in ranges of MIN_RANGE levels at the least (on average, rounded up).
// Otherwise the last, partly filled wave is: what is left after the full
// waves, or that and one full wave more.  There the extra work counts too, as
// another launch beside this one may fill the idle SMs: a range more has to
// shorten the launch by EXTRA times what it adds to the work of an SM, and the
// launch is never longer than one cut as a whole.
//
// Steps in fast arithmetic, all columns cut or none -> this rule: 96x250x35 with
// 7 species (168 tiles on 148 SMs) 222 -> 198 us, 512x400x40 with one (171) 329
// -> 283, 256x256x40 with 5 (300) 400 -> 333, 250x210x40 with 12 (600) 688 ->
// 594, 512x26x40 with 12 (216) 242 -> 226; 187x301x33 with 5 (280) 277, not cut,
// and 128x128x20 with one (18) 41, cut as a whole, either way.  Without EXTRA
// 96x250x35 takes 179, and three handles stepping 164x279x43 with 8 species
// beside each other 3 % longer than with no cut (with it 1 %).
#pragma once

namespace icar {
namespace op {

constexpr int MIN_RANGE = 5, EXTRA = 5;

struct ColumnSplit {
    long whole;
    int parts;
};

// First level of range k.  The march of the lowest range starts at the ground,
// the others' two levels below their own, where they do less than half of a
// level's work: the lowest has a level more (9 levels: 5 and 4, where 4 and 5
// took 46 us instead of 43 for a step of 19x116x9).
#ifdef __CUDACC__
__host__ __device__
#endif
inline int range_begin(int nz, int parts, int k) { return k == 0 ? 0 : (nz - 1) * k / parts + 1; }

// levels an SM marches, one after the other, for `tiles` tiles of nz levels in
// `parts` ranges each
inline int range_cost(int nz, int parts) { return (nz + parts - 1) / parts + 2 + (parts > 1 ? 3 : 0); }
inline long march_cost(long tiles, int nz, int parts, int sms)
{
    return (tiles * parts + sms - 1) / sms * range_cost(nz, parts);
}
inline bool can_cut(int nz, int parts) { return (nz + parts - 1) / parts >= MIN_RANGE; }

// all columns cut alike
inline int best_parts(long tiles, int nz, int sms)
{
    int best = 1;
    for (int n = 2; can_cut(nz, n); n++)
        if (march_cost(tiles, nz, n, sms) < march_cost(tiles, nz, best, sms)) best = n;
    return best;
}

inline ColumnSplit split_columns(long tiles, int nz, int sms)
{
    auto length = [&](const ColumnSplit &s) {
        return march_cost(s.whole, nz, 1, sms) + march_cost(tiles - s.whole, nz, s.parts, sms);
    };
    // length of the launch and EXTRA times its work, in levels x SMs
    auto cost = [&](const ColumnSplit &s) {
        return length(s) * sms +
               EXTRA * (s.whole * range_cost(nz, 1) + (tiles - s.whole) * s.parts * range_cost(nz, s.parts));
    };
    const ColumnSplit all{0, best_parts(tiles, nz, sms)};
    ColumnSplit best = all;
    for (long whole = tiles / sms * sms, n = 0; whole > 0 && n < 2; whole -= sms, n++)
        for (int parts = 1; parts == 1 || can_cut(nz, parts); parts++) {
            const ColumnSplit s{whole, parts};
            if (length(s) <= length(all) && cost(s) < cost(best)) best = s;
        }
    return best;
}

// CTAs of the launch, and the tile and level range [ka, kb) of CTA b (tiles are
// counted with the species fastest)
inline long split_ctas(const ColumnSplit &s, long tiles) { return s.whole + (tiles - s.whole) * s.parts; }
#ifdef __CUDACC__
__host__ __device__
#endif
inline void split_cta(unsigned b, unsigned whole, int parts, unsigned species, int nz, unsigned &tile, int &ka, int &kb)
{
    if (b < whole) {
        tile = b, ka = 0, kb = nz;
        return;
    }
    // the ranges of a column side by side (they share levels in L2), those of a
    // launch cut as a whole by species (which share the winds' planes)
    unsigned q = b - whole, k;
    if (whole == 0) {
        const unsigned s = q % species;
        q /= species;
        k = q % (unsigned)parts;
        tile = q / (unsigned)parts * species + s;
    } else {
        k = q % (unsigned)parts;
        tile = whole + q / (unsigned)parts;
    }
    ka = range_begin(nz, parts, (int)k);
    kb = range_begin(nz, parts, (int)k + 1);
}

}  // namespace op
}  // namespace icar
