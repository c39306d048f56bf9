"""The running sums of the sampler's warps (turkce_llm_b200/csrc/lane_scan.h) over an array of 32 lanes on the CPU."""
from conftest import compile_and_run

CHECK = r"""
#include "lane_scan.h"
#include <cmath>
#include <cstdio>
#include <random>
struct Lanes { double v[32]; };
int main() {
    std::mt19937_64 rng(1);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    long backwards = 0, plain_backwards = 0, off = 0;
    for (int trial = 0; trial < 200000; ++trial) {
        // sums of exponentials of logits over a wide range: many shares are around the last bit of the running sum or zero
        Lanes x;
        for (double& v : x.v) v = u(rng) < 0.2 ? 0.0 : (double)expf((float)(-45.0 * u(rng)));
        auto add = [](Lanes a, int o) { for (int l = 31; l >= o; --l) a.v[l] = a.v[l] + a.v[l - o]; return a; };
        auto max = [](Lanes a, int o) { for (int l = 31; l >= o; --l) a.v[l] = std::fmax(a.v[l], a.v[l - o]); return a; };
        auto keep = [](Lanes a, int) { return a; };
        const Lanes plain = tb::monotone_lane_sums(x, add, keep), m = tb::monotone_lane_sums(x, add, max);
        double exact = 0.0;
        for (int l = 0; l < 32; ++l) {
            exact += x.v[l];
            if (l > 0 && plain.v[l] < plain.v[l - 1]) ++plain_backwards;
            if (l > 0 && m.v[l] < m.v[l - 1]) ++backwards;
            if (!(std::fabs(m.v[l] - exact) <= 64 * 0x1p-53 * exact)) ++off;        // at most 31 + 31 roundings
        }
    }
    printf("%ld steps back, %ld without the maximum, %ld sums off\n", backwards, plain_backwards, off);
    return backwards != 0 || plain_backwards == 0 || off != 0;
}
"""


def test_lane_sums_never_go_backwards(tmp_path):
    """(and do without the maximum, on the same values: the inputs reach the case)"""
    print(compile_and_run(tmp_path, CHECK))
