// set_j between firsthalf and lasthalf waits for the copy of the staged
// updates that went with the call, not for its forces or results.  Run by
// tests/test_engine_host.py.
#include "engine_host.h"

using namespace g6;

int main() {
    int bad = 0;
    const double zero[3] = {0, 0, 0};
    static int idx[200];
    static double x[200][3], v[200][3], acc[200][3], jerk[200][3], pot[200];
    static int nn[200];
    Engine e(0);
    e.set_npipes(200);
    for (int round = 0; round < 3; ++round) {
        for (int j = 0; j < 100; ++j) bad += e.set_j(j, j, 0.0, 1.0, nullptr, zero, zero, zero, zero) != 0;
        e.set_ti(1.0 + round);
        fake::waited_for = 0;
        bad += e.firsthalf(100, 200, idx, x, v, 0.0, nullptr) != 0;
        for (int j = 0; j < 50; ++j) bad += e.set_j(j, j, 0.0, 2.0, nullptr, zero, zero, zero, zero) != 0;
        if (fake::waited_for >= fake::force_at || fake::scatters != round + 1) {
            std::printf("set_j waited for operation %lld; the forces are %lld\n", fake::waited_for, fake::force_at);
            ++bad;
        }
        bad += e.lasthalf(200, acc, jerk, pot, nn) != 0;
        if (pot[0] != 100.0) {  // the call's own j-state
            std::printf("pot %g\n", pot[0]);
            ++bad;
        }
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
