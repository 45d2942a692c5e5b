// Checks of hicar_b200/csrc/launch_split.h: the CTAs of a launch cover every
// level of every tile once, in ranges of at least MIN_RANGE levels where a
// column is cut, equal to one level; and a launch is never longer than its full
// waves followed by what is left as a launch of its own.  Exit status 1 on any
// failure.
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
                bad += s.whole < 0 || s.whole > tiles || s.whole % sms != 0 || s.parts < 1 || n < tiles;
                std::vector<int> next(tiles, 0), least(tiles, nz), most(tiles, 0);
                std::vector<int> at(tiles * (long)nz, 0);
                for (long b = 0; b < n; b++) {
                    unsigned tile;
                    int ka, kb;
                    split_cta((unsigned)b, (unsigned)s.whole, s.parts, (unsigned)tiles, nz, tile, ka, kb);
                    if (tile >= tiles || ka < 0 || kb > nz || ka >= kb) {
                        bad++;
                        continue;
                    }
                    for (int k = ka; k < kb; k++) at[tile * (long)nz + k]++;
                    if (kb - ka < least[tile]) least[tile] = kb - ka;
                    if (kb - ka > most[tile]) most[tile] = kb - ka;
                }
                for (int c : at) bad += c != 1;
                for (long t = 0; t < tiles; t++) bad += most[t] - least[t] > 1 || (least[t] < nz && least[t] < MIN_RANGE);
                auto cost = [&](const ColumnSplit &x, long t) {
                    return march_cost(x.whole, nz, 1, sms) + march_cost(t - x.whole, nz, x.parts, sms);
                };
                const long full = tiles / sms * sms, rest = tiles - full;
                const long apart = march_cost(full, nz, 1, sms) + (rest ? march_cost(rest, nz, best_parts(rest, nz, sms), sms) : 0);
                bad += cost(s, tiles) > apart;
                checked++;
            }
    std::printf("checked=%ld failures=%ld\n", checked, bad);
    return bad != 0;
}
