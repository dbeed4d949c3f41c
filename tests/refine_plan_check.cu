// refine_plan_check.cu -- host-only check of the plan that the mixed mode's
// FP64 refinement runs (refine_config, refine_tasks and batch_plan in
// starlab_b200/csrc/kernels.h), built and run by tests/test_refine_plan.py
// without a GPU.
//
// For every number of flagged particles of calls from 1 to 2^20, j-counts up
// to 2^20 and resident CTAs of one to four per SM: the splits' partials fit
// the buffer the call has (refine_partial_records), the i-tiles its counters
// (one per i of the call), the splits cover the padded j-set without an empty
// one; and from one wave of tasks up, the last wave is no emptier than the
// plan without the rule would leave it.
#include <cstdio>
#include <vector>
#include "kernels.h"

using namespace g6;

static ForceParams plan(ForceConfig c, int tasks, int count, int nj, int nj_pad, int &nt) {
    ForceParams p{};
    p.ni = count;
    p.nj = nj;
    p.nj_pad = nj_pad;
    c.nsplit = tasks;
    batch_plan(kKernF64, c, p, nt);
    return p;
}

int main() {
    std::vector<int> sizes;
    for (int v = 1; v <= (1 << 20); v = v < 8 ? v + 1 : v + v / 3) sizes.push_back(v);
    for (int v : {31, 32, 33, 63, 64, 65, 78, 127, 128, 129, 4818, 16384, 65536, 262144}) sizes.push_back(v);
    ForceConfig batch{32, 1, 8, 4, 0};
    const ForceConfig c = refine_config(batch);
    long long checked = 0, waves = 0;
    for (int slots : {148, 296, 444, 592})
        for (int nj : sizes) {
            const int T = tile_of(kKernF64), nj_pad = (nj + T - 1) / T * T;
            for (int count : sizes)
                for (int calls_ni : {count, 2 * count, 40 * count}) {
                    if (calls_ni > (1 << 20)) continue;
                    int nt = 0;
                    const ForceParams p = plan(c, refine_tasks(c, count, calls_ni, nj_pad, slots), count, nj, nj_pad, nt);
                    const int itile = batch_item_itile(kKernF64, c, count), n_itiles = (count + itile - 1) / itile;
                    const char *bad = nullptr;
                    if ((size_t)p.nsplit * count > refine_partial_records(calls_ni)) bad = "partials";
                    if (n_itiles > calls_ni) bad = "counters";
                    if ((long long)p.nsplit * p.jper < nj_pad || (long long)(p.nsplit - 1) * p.jper >= nj_pad ||
                        p.jper % T)
                        bad = "splits do not tile the j-set";
                    if (nt != n_itiles * p.nsplit) bad = "task count";
                    int old_nt = 0;
                    plan(c, refine_tasks_wanted(count, nj_pad), count, nj, nj_pad, old_nt);
                    if (nt >= slots && old_nt >= slots) {
                        ++waves;
                        const auto fill = [&](int t) { return (double)t / (((t + slots - 1) / slots) * (long long)slots); };
                        // (within one j-tile of rounding, and never under the 94 % that the rule stops at)
                        if (fill(nt) < 0.94 && fill(nt) < fill(old_nt) - 0.06) bad = "an emptier last wave";
                    }
                    if (bad) {
                        std::printf("%s: slots %d nj %d count %d calls_ni %d: nsplit %d jper %d tasks %d (%d)\n", bad, slots,
                                    nj, count, calls_ni, p.nsplit, p.jper, nt, old_nt);
                        return 1;
                    }
                    ++checked;
                }
        }
    std::printf("ok %lld %lld\n", checked, waves);
    return 0;
}
