// column_split_check.cu -- host program: whatever cut column_split chooses, segment_levels hands
// every level of a column to exactly one segment, in order, with no empty segment.
#include <cstdio>

#include "mg_common.cuh"

int main()
{
    int n = 0, cut = 0, bad = 0;
    for (long long tiles = 1; tiles <= 1200; tiles = tiles < 80 ? tiles + 1 : tiles + 37)
        for (int nz = 1; nz <= 320; nz = nz < 40 ? nz + 1 : nz + 13)
            for (int per_sm = 1; per_sm <= 2; per_sm++)
                for (double lead : {1.5, 2.5, 3.}) {
                    const ColSplit c = column_split(tiles, nz, per_sm, lead);
                    int prev = 0;
                    for (int s = 0; s < c.nseg + c.ns; s++) {
                        int kb, ke;
                        segment_levels(nz, c.nseg, c.ns, c.ls, s, kb, ke);
                        if (kb != prev + 1 || ke < kb) bad++;
                        prev = ke;
                    }
                    if (prev != nz || c.nseg < 1) bad++;
                    n++;
                    cut += c.ns > 0;
                }
    printf("%d grids, %d with short segments, %d wrong\n", n, cut, bad);
    return bad != 0 || cut == 0;
}
