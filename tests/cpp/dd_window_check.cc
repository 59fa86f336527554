// Host check of the distance-driven grad's staged window (dd_window.h): for
// every reach and tile extent that the tiles take, every piece that is formed
// reads staged channels only, and every piece that a position of the tile falls
// in is formed.  Prints the number of windows and of failures.
#include <cmath>
#include <cstdio>

#include "../../ct_recon_extensions_gb300/csrc/dd_window.h"

using namespace ctr;

int main()
{
    int cases = 0, bad = 0;
    for (int re = 0; re < 64 * 16; ++re)
        for (int ex = 0; ex < 64 * 16; ++ex) {
            const float reach = re / 16.0f, e = 0.51f + ex / 16.0f;
            if (!dg_fits(e, reach)) continue;
            ++cases;
            const int need = dg_need(e, reach), m = dg_spread(static_cast<long long>(2.0 * reach * 4294967296.0));
            const int first = dg_first_piece(need, m), end = kDgHalf + need;
            bool ok = first - m >= 0 && end <= 2 * kDgHalf;  // reads [first - m, end], one zero behind the channels
            // positions y = x + reach - 1 with |x| <= e round to pieces; a hair more for the FP32 positions
            const double lo = -e + reach - 1.0 - 1e-4, hi = e + reach - 1.0 + 1e-4;
            ok = ok && kDgHalf + std::floor(lo + 0.5) >= first && kDgHalf + std::ceil(hi - 0.5) < end;
            bad += !ok;
        }
    std::printf("%d %d\n", cases, bad);
    return 0;
}
