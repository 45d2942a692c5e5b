// Checks of hicar_b200/csrc/launch_split.h: the CTAs of a launch cover every
// level of every tile once, in ranges equal to one level (the lowest has one more)
// and no shorter than MIN_RANGE allows; and a cut launch is never longer than one of
// whole columns.  Exit status 1 on any failure.
#include <cstdio>
#include <vector>

#include "../hicar_b200/csrc/launch_split.h"

using namespace icar::op;

int main()
{
    long bad = 0, checked = 0;
    for (int sms : {1, 7, 148})
        for (long tiles = 1; tiles <= 1000; tiles += tiles < 320 ? 1 : 37)
            for (int nz : {1, 2, 3, 4, 5, 9, 10, 11, 20, 21, 33, 46, 60}) {
                const ColumnSplit s = split_columns(tiles, nz, sms);
                const long n = split_ctas(s, tiles);
                const unsigned species = tiles % 5 == 0 ? 5 : tiles % 3 == 0 ? 3 : 1;
                bad += s.whole < 0 || s.whole > tiles || s.whole % sms != 0 || s.parts < 1 || n < tiles;
                std::vector<int> least(tiles, nz + 1), most(tiles, 0);   // a tile's shortest and longest range
                std::vector<int> at(tiles * (long)nz, 0);
                for (long b = 0; b < n; b++) {
                    unsigned tile;
                    int ka, kb;
                    split_cta((unsigned)b, (unsigned)s.whole, s.parts, species, nz, tile, ka, kb);
                    if (tile >= tiles || ka < 0 || kb > nz || ka >= kb) {
                        bad++;
                        continue;
                    }
                    for (int k = ka; k < kb; k++) at[tile * (long)nz + k]++;
                    const int march = kb - ka + (ka ? 1 : 0);
                    if (march < least[tile]) least[tile] = march;
                    if (march > most[tile]) most[tile] = march;
                }
                for (int c : at) bad += c != 1;
                for (long t = 0; t < tiles; t++) bad += most[t] - least[t] > 1;
                bad += s.parts > 1 && (nz + s.parts - 1) / s.parts < MIN_RANGE;
                auto length = [&](const ColumnSplit &x) {
                    return march_cost(x.whole, nz, 1, sms) + march_cost(tiles - x.whole, nz, x.parts, sms);
                };
                bad += length(s) > length({0, 1});
                checked++;
            }
    std::printf("checked=%ld failures=%ld\n", checked, bad);
    return bad != 0;
}
