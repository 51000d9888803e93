// C entry points over the activity kernels' shared arithmetic (rl_math.cuh)
// for tests/test_activity_math_host.py.
#include "../../relearn_b200/csrc/rl_math.cuh"

extern "C" {
// entries of q whose 2 exp(-q) - 1 differs in its bits from the step-by-step form
long probe_curve(long n, const double* q) {
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        const double a = rl::rl_two_exp_minus_one(q[i]);
        const double b = rl::rl_fma(2.0, rl::rl_exp(-q[i]), -1.0);
        bad += !(rl::as_u64(a) == rl::as_u64(b) || (a != a && b != b));
    }
    return bad;
}
// entries of b (53 random bits) whose uniform, or whose piece of the normal
// quantile, differs from the formulas with conversions and FP64 comparisons
long probe_uniform(long n, const unsigned long long* b) {
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        const double p = ((double)b[i] + 0.5) * 1.1102230246251565404e-16;
        const double got = rl::uniform_from_bits53(b[i]);
        bad += rl::as_u64(got) != rl::as_u64(p) || rl::normal_in_tail(got) != !(__builtin_fabs(p - 0.5) <= 0.425);
    }
    return bad;
}
}
