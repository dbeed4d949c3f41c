// Opening an engine prepares no one-launch kernel; a kind of small call
// prepares its own the first time, once per open engine.  Run by
// tests/test_engine_host.py.
#include "engine_host.h"

using namespace g6;

int main() {
    int bad = 0;
    const double zero[3] = {0, 0, 0};
    int idx[1] = {0}, nn[1];
    double x[1][3] = {}, v[1][3] = {}, acc[1][3], jerk[1][3], pot[1], h2[1] = {1.0};
    auto expect = [&](const char *when, int want) {
        if (fake::prepared != want) std::printf("%s: %d prepared, not %d\n", when, fake::prepared, want), ++bad;
    };
    Engine e(0);
    for (int opened = 0; opened < 2; ++opened) {
        bad += e.open(0, 0) != 0;
        expect("open", 2 * opened);
        for (int k = 0; k < 4; ++k) {
            bad += e.set_j(0, 0, 0.0, 1.0, nullptr, zero, zero, zero, zero) != 0;
            bad += e.firsthalf(1, 1, idx, x, v, 0.0, k & 1 ? h2 : nullptr) != 0;
            bad += e.lasthalf(1, acc, jerk, pot, nn) != 0;
            expect("call", 2 * opened + std::min(k + 1, 2));
        }
        e.close();
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
