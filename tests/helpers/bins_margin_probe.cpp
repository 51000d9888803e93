// C entry points over the FP32 search's certified margin (rl_math.cuh) for
// tests/test_bins_margin_host.py.
#include "../../relearn_b200/csrc/rl_math.cuh"

extern "C" {
double probe_margin(double total, unsigned visited) { return rl::bins_margin32(total, visited); }
// the compensated sum as the FP32 searches run it
float probe_kahan(long n, const float* x) {
    float s = 0.0f, c = 0.0f;
    for (long i = 0; i < n; ++i) {
        const float y = x[i] - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    return s;
}
}
