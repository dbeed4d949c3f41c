// A status word that a failed call left behind does not reach a later call:
// the two words are used in turn, each cleared by the call before, and a
// call that fails on the host clears nothing.  Run by tests/test_engine_host.py.
#include "engine_host.h"

using namespace g6;

int main() {
    int bad = 0;
    const double zero[3] = {0, 0, 0};
    static int idx[100];
    static double x[100][3], v[100][3], acc[100][3], jerk[100][3], pot[100];
    static int nn[100];
    for (int ni : {100, 1}) {  // 1: with an update, the small-call forms
        for (int fits : {1, 0}) {
            fake::small_fits = fits;
            fake::nsplit = 1;
            Engine e(0);
            e.set_npipes(100);
            auto call = [&](double m) {
                e.set_j(0, 0, 0.0, m, nullptr, zero, zero, zero, zero);
                const int rc = e.firsthalf(1, ni, idx, x, v, 0.0, nullptr);
                return rc ? rc : e.lasthalf(ni, acc, jerk, pot, nn);
            };
            bad += call(1.0) != 0;
            fake::report = ST_TMA_TIMEOUT;  // a call whose copy wait ran out
            const int rc = call(2.0);
            const bool one = ni == 1 && fits;  // has no copy waits, brings no status back
            if (rc != (one ? 0 : 3)) std::printf("reported: %d\n", rc), ++bad;
            fake::fail_force = true;
            if (call(3.0) == 0) std::printf("the failed launch was not reported\n"), ++bad;
            for (int k = 0; k < 3; ++k) {
                const int later = call(4.0 + k);
                if (later || pot[0] != 4.0 + k) std::printf("ni %d: a later call returned %d, %g\n", ni, later, pot[0]), ++bad;
            }
        }
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
