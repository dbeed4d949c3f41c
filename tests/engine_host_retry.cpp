// A call repeated in a wider fixed-point range takes the j-updates it had:
// those that set_j has staged since firsthalf, however many, are the next
// call's.  Run by tests/test_engine_host.py.
#include "engine_host.h"

using namespace g6;

int main() {
    int bad = 0;
    const double zero[3] = {0, 0, 0};
    constexpr int N = 3 * kSmallMax;
    for (int later : {1, kSmallMax, N}) {  // updates staged beside the running call
        fake::small_fits = 0;
        fake::nsplit = 1;
        Engine e(0);
        auto set = [&](int a, double m) { return e.set_j(a, a, 0.0, m, nullptr, zero, zero, zero, zero); };
        static int idx[1], nn[1];
        static double x[1][3], v[1][3], acc[1][3], jerk[1][3], pot[1];
        auto first = [&] { return e.firsthalf(N, 1, idx, x, v, 0.0, nullptr); };
        auto last = [&] { return e.lasthalf(1, acc, jerk, pot, nn); };
        for (int j = 0; j < N; ++j) bad += set(j, 1.0) != 0;
        e.set_ti(1.0);
        bad += first() != 0 || last() != 0;
        bad += set(0, 2.0) != 0;  // with one update the small-call form
        const int small = fake::small_calls;
        fake::report = ST_RANGE;
        bad += first() != 0;
        if (fake::small_calls != small + 1) std::printf("not the small-call form\n"), ++bad;
        for (int j = 0; j < later; ++j) bad += set(j, 3.0) != 0;
        const int calls = fake::force_calls;
        bad += last() != 0;
        if (fake::force_calls != calls + 1) std::printf("not repeated\n"), ++bad;
        if (pot[0] != N + 1) std::printf("%d staged: the call's j-state sums to %g\n", later, pot[0]), ++bad;
        bad += first() != 0 || last() != 0;
        if (pot[0] != N + 2 * later) std::printf("%d staged: the next call's sums to %g\n", later, pot[0]), ++bad;
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
