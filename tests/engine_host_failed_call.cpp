// A small FP64 call that fails between taking its j-updates and its launch
// (no memory for the split partials; a refused launch) keeps them: the next
// call at the same time sees the updated particle.  Run by
// tests/test_engine_host.py.
#include "engine_host.h"

using namespace g6;

namespace {
const double zero[3] = {0, 0, 0};
int set(Engine &e, int a, double m) { return e.set_j(a, a, 0.0, m, nullptr, zero, zero, zero, zero); }
int call(Engine &e, int nj, int ni, double *pot) {
    int idx[64] = {};
    double x[64][3] = {}, v[64][3] = {}, acc[64][3], jerk[64][3];
    int nn[64];
    const int rc = e.firsthalf(nj, ni, idx, x, v, 0.0, nullptr);
    return rc ? rc : e.lasthalf(ni, acc, jerk, pot, nn);
}
int expect(const char *what, double got, double want) {
    if (got == want) return 0;
    std::printf("%s: %g, not %g\n", what, got, want);
    return 1;
}
}  // namespace

int main() {
    int bad = 0;
    for (int fits : {1, 0})       // one launch; updates and prediction, then forces
        for (int how : {0, 1}) {  // the partials' cudaMalloc, the force launch
            fake::small_fits = fits;
            fake::nsplit = 1;
            Engine e(0);
            double pot[64];
            for (int j = 0; j < 3; ++j) bad += set(e, j, 1.0) != 0;
            e.set_ti(1.0);
            bad += call(e, 3, 1, pot) != 0;
            bad += expect("before", pot[0], 3.0);
            bad += set(e, 1, 5.0) != 0;
            fake::nsplit = 8;  // the call needs partials it has not got
            if (how)
                fake::fail_force = true;
            else
                fake::fail_malloc = 0;
            bad += call(e, 3, 1, pot) == 0;
            fake::fail_malloc = -1;
            fake::fail_force = false;
            bad += call(e, 3, 1, pot) != 0;
            bad += expect("after the failed call", pot[0], 7.0);
            bad += set(e, 1, 2.0) != 0;
            bad += call(e, 3, 1, pot) != 0;
            bad += expect("a later update", pot[0], 4.0);
        }
    if (!bad) std::printf("ok\n");
    return bad;
}
