// Host-side check of the cap gather's choice of form (csrc/gather_smem.cuh): for
// every volume size, cap band and angle count that a context accepts, a form is
// chosen whose dynamic and static shared memory fit a CTA.  Runs no GPU code.
#include <cstdio>

#include "gather_smem.cuh"

using namespace tdm;

int main() {
    long long checked = 0, wide = 0;
    for (int D = 128; D <= 1024; D *= 2) {
        const int F = D / 2;  // the largest field: a band has at most sqrt(2) F + 2 planes
        for (int band = 1; band <= (int)(1.41422 * F) + 2; ++band)
            for (int n = 1; n <= 65535 && gather_limit_bytes(D, band, n) <= kMaxSmemPerCta; ++n)
                for (int counts = 0; counts < 2; ++counts) {
                    const int w = gather_columns(D, band, n, counts);
                    const size_t used = w == 16  ? GatherSmem<16>::bytes(band, n) + sizeof(unsigned[2][32])
                                        : w == 8 ? GatherSmem<8>::bytes(band, n) + sizeof(unsigned[2][32])
                                                 : ~size_t(0);
                    if (used > 232448) {
                        std::printf("D %d band %d n %d counts %d: %d columns, %zu bytes\n", D, band, n, counts, w, used);
                        return 1;
                    }
                    wide += w == 16;
                    ++checked;
                }
    }
    std::printf(checked > 1000000 && wide > 0 ? "ok\n" : "too few\n");
    return 0;
}
