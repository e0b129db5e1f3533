// mhh_fft_plan.h -- the stages of the run-time-plan transforms (mhh_pres.cu) per
// length; plain C++.
#pragma once

#include <algorithm>
#include <vector>

namespace mhh
{
    // The radices (2 to 10) of the run-time plan: the fewest factors, and of
    // those the smallest sum (the least arithmetic), larger ones first.
    inline int plan_radices(int n, int* fac)
    {
        std::vector<int> divs, best, pick;      // divisors of n, best radix of each
        for (int d=1; d<=n; ++d) if (n % d == 0) divs.push_back(d);
        best.assign(divs.size(), 1 << 20);
        pick.assign(divs.size(), 0);
        best[0] = 0;
        for (size_t a=1; a<divs.size(); ++a)
            for (int r=2; r<=10; ++r)
                if (divs[a] % r == 0)
                {
                    const size_t b = std::lower_bound(divs.begin(), divs.end(), divs[a]/r) - divs.begin();
                    const int cost = best[b] + 64 + r;
                    if (cost < best[a]) { best[a] = cost; pick[a] = r; }
                }
        int nfac = 0;
        for (int d = n; d > 1; )
        {
            const size_t a = std::lower_bound(divs.begin(), divs.end(), d) - divs.begin();
            fac[nfac++] = pick[a];
            d /= pick[a];
        }
        std::sort(fac, fac + nfac, [](int x, int y) { return x > y; });
        return nfac;
    }

    // The stage codes RA + 16 RB of the float plan; the elementary radices of a
    // length fix the rounding of its transforms (see fe_stage).  Radix 8 after 2,
    // 4 or 8 in frequency (RB = 0) at 128, 256 and 512; radices 8, 4, 2, 3 at the
    // nine lengths listed, which had stages of radix 8 before there was a plan;
    // radices 4, 2, 3, 5, 7 at every other length, 1536 and 2048 among them.
    // Neighbours are grouped where there is a stage of the product.
    inline int plan_floats(int n, int* fac)
    {
        if (n == 128 || n == 256 || n == 512)
        {
            fac[0] = n/64; fac[1] = fac[2] = 8;
            return 3;
        }
        int nfac = 0;
        bool eights = false;
        for (int m : {16, 32, 48, 64, 96, 192, 384, 768, 1024}) eights = eights || n == m;
        std::vector<int> rad;
        int r = n;
        for (int f : {8, 4, 2, 3, 5, 7})
            while ((f < 8 || eights) && r % f == 0) { rad.push_back(f); r /= f; }
        for (size_t q=0; q<rad.size(); ++q)
        {
            int code = rad[q] + 16;
            if (q + 1 < rad.size())
                for (int pair : {0x32, 0x52, 0x24, 0x33, 0x34})
                    if (rad[q] == (pair & 15) && rad[q+1] == pair >> 4) { code = pair; ++q; break; }
            fac[nfac++] = code;
        }
        return nfac;
    }
}
