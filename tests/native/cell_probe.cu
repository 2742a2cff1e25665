// Host check of fx_cell64 (csrc/qew_fix.cuh) against the reference's fold
// (filtered_noise.h:80-92) in FP64: reads "a n" pairs of hexadecimal bits and
// decimal periods for k = 0 from stdin, prints the pairs that were accepted with
// another cell or fraction, and last the counts of accepted and declined.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "../../qew_gb300/csrc/qew_fix.cuh"

int main() {
    unsigned long long bits;
    int n;
    long accepted = 0, declined = 0, wrong = 0;
    while (scanf("%llx %d", &bits, &n) == 2) {
        double g;
        memcpy(&g, &bits, sizeof(g));
        int iy = -1;
        unsigned long long f = 0;
        if (!fx_cell64(g, 0, n, iy, f)) {
            ++declined;
            continue;
        }
        ++accepted;
        const double nd = (double)n;
        double r = g;
        if (!(r >= 0.0 && r < nd)) r -= std::floor(r / nd) * nd;
        int ix = (int)std::floor(r);
        if (ix >= n) {
            ix -= n;
            r -= nd;
        }
        const double fx = r - (double)ix;
        const unsigned long long want = (unsigned long long)std::ldexp(fx, 64);
        if (ix != iy || want != f) {
            ++wrong;
            printf("wrong %a n %d: cell %d fraction %llx, reference %d %llx\n", g, n, iy, f, ix, want);
        }
    }
    printf("accepted %ld declined %ld wrong %ld\n", accepted, declined, wrong);
    return wrong ? 1 : 0;
}
