// Host check of the single-view walk's addresses (sv_walk.h), built with signed
// overflow trapping: for both directions and every channel of rows anywhere in
// shared memory, the address that the walk forms from a position's number is the
// channel's.  Prints the number of cases and of failures.
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "../../ct_recon_extensions_gb300/csrc/sv_walk.h"

using namespace ctr;

int main()
{
    int cases = 0, bad = 0;
    for (unsigned at : {0u, 1024u, 232000u})
        for (int dir4 : {4, -4})
            for (int i0 = 1; i0 < 4000; i0 += 7)
                for (int r = -70; r <= 70; ++r) {
                    // r channels along the walk from the reference: channel c before, n after the position
                    const int c = dir4 > 0 ? i0 + r : i0 + 1 - r, n = c + dir4 / 4;
                    if (n < 0) continue;
                    const float f = 12582912.0f + r;
                    int num;
                    std::memcpy(&num, &f, sizeof num);
                    ++cases;
                    bad += sv_address(sv_base(at, dir4 > 0 ? i0 : i0 + 1, dir4), num, dir4) != at + 4u * n;
                }
    std::printf("%d %d\n", cases, bad);
    return 0;
}
