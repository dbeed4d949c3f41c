// An allocation that fails while a call's buffers grow leaves no capacity
// behind that the buffers no longer have: the next call allocates what it
// needs.  Run by tests/test_engine_host.py.
#include "engine_host.h"

using namespace g6;

int main() {
    int bad = 0;
    const double zero[3] = {0, 0, 0};
    static int idx[600];
    static double x[600][3], v[600][3], acc[600][3], jerk[600][3], pot[600], h2[600];
    static int nn[600];
    for (int k = 0; k < 600; ++k) h2[k] = 1.0;
    for (int nb : {0, 1})
        for (int which = 0; which < 8; ++which) {  // the allocation that fails (of d_irec_ up to the lists' offsets)
            fake::nsplit = 4;
            Engine e(0);
            e.set_npipes(600);
            for (int j = 0; j < 3; ++j) bad += e.set_j(j, j, 0.0, 1.0, nullptr, zero, zero, zero, zero) != 0;
            e.set_ti(1.0);
            auto call = [&](int ni) {
                const int rc = e.firsthalf(3, ni, idx, x, v, 0.0, nb ? h2 : nullptr);
                return rc ? rc : e.lasthalf(ni, acc, jerk, pot, nn);
            };
            e.set_npipes(70);
            bad += call(70) != 0;
            e.set_npipes(600);
            fake::nsplit = 16;
            fake::fail_malloc = which;
            const bool failed = call(600) != 0;
            if (nb) e.read_neighbours();  // whatever it answers, from buffers that are there
            fake::fail_malloc = -1;
            fake::nsplit = 4;
            const bool again = call(70) != 0 || call(600) != 0;  // would use freed or null buffers
            if (again || pot[599] != 3.0) {
                std::printf("nb %d allocation %d (failed %d): the next call does not work\n", nb, which, failed);
                ++bad;
            }
        }
    if (!bad) std::printf("ok\n");
    return bad;
}
