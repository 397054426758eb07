// Host build of the step controller (cosmos_gb300/csrc/device_common.cuh): a run whose steps are taken in any
// order by the two forms that share it -- the time step kernel with sweeps that reduce into the next slot, and the
// fused step, whose last block enters the step after the reduction -- forms every time step from the maximum of
// the step before alone.  Speeds fall from step to step, so that a value left over from an earlier step would
// win.  Prints what differs; exits non-zero if anything does.
#include "cuda_runtime.h"

#include <cstdio>

#include "../../cosmos_gb300/csrc/device_common.cuh"

using namespace cg;

static void reduce(unsigned long long* slot, double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (b > *slot) *slot = b;
}

int main() {
    constexpr int kSteps = 10;
    long differ = 0;
    for (int order = 0; order < 1 << kSteps; order++) {
        StepCtl c;
        memset(&c, 0, sizeof c);
        c.t_final = 1e30;
        c.cfl = 0.9;
        c.dx = 0.01;
        c.it_limit = kSteps;
        c.active = 1;
        double speed = 4.0;
        reduce(&c.smax[0], speed);
        for (int k = 0; k < kSteps; k++) {
            double want = 0.9 * (0.01 / speed);
            if (k <= 5) want = want * 0.2;
            speed *= 0.9;
            if (order >> k & 1) {  // the fused step
                const StepNow s = step_now(&c);
                const int it = c.it;
                reduce(&c.smax[(it + 1) & 1], speed);
                step_enter(&c, s, it & 1);
            } else {
                step_ctl_advance(&c);
                reduce(&c.smax[c.it & 1], speed);
            }
            if (c.dt != want && differ++ < 10) printf("forms %x, step %d: dt %a, not %a\n", order, k, c.dt, want);
        }
    }
    printf("%ld differ\n", differ);
    return differ != 0;
}
