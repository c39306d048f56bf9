"""The helper threads of large host copies (turkce_llm_b200/csrc/copy_helpers.h), on the CPU."""
from conftest import compile_and_run

CHECK = r"""
#include "copy_helpers.h"
#include <cstdio>
#include <cstdlib>
#include <sys/wait.h>
int main() {
    // every slot runs once per job, from the first to the thousandth
    for (int job = 0; job < 1000; ++job) {
        std::atomic<int> ran[tb::kHelperSlots] = {};
        tb::helpers().run([&](int t) { ran[t].fetch_add(1); });
        for (auto& r : ran)
            if (r.load() != 1) { printf("job %d: a slot ran %d times\n", job, r.load()); return 1; }
    }
    // a child forked now has none of the threads: it still runs a job (by itself), and leaves by exit
    for (int use = 0; use < 2; ++use) {
        fflush(stdout);
        const pid_t child = fork();
        if (child == 0) {
            int ran = 0;
            if (use) tb::helpers().run([&](int) { ++ran; });
            exit(use && ran != tb::kHelperSlots ? 3 : 0);
        }
        int status = 0;
        waitpid(child, &status, 0);
        if (!WIFEXITED(status) || WEXITSTATUS(status) != 0) { printf("child: status %#x\n", status); return 1; }
    }
    // threads can be given back, and come again
    tb::helpers().stop();
    std::atomic<int> ran{0};
    tb::helpers().run([&](int) { ++ran; });
    return ran.load() == tb::kHelperSlots ? 0 : 1;
}
"""


def test_helpers_run_every_slot_and_survive_a_fork(tmp_path):
    compile_and_run(tmp_path, CHECK, "-pthread")


HANDOUT = r"""
#include "copy_helpers.h"
#include <cstdio>
#include <vector>
int main() {
    tb::Handout<12> h;
    int a[12], b[12], c[12];
    // what one holder keeps, others do without: nobody waits
    if (h.take(4, a) != 4 || h.take(12, b) != 8 || h.take(1, c) != 0) { printf("counts\n"); return 1; }
    h.give(a, 4);
    if (h.take(12, c) != 4) { printf("given back\n"); return 1; }
    h.give(b, 8);
    h.give(c, 4);
    // nothing is held twice at a time
    std::atomic<int> held[12] = {};
    std::atomic<bool> twice{false};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int i = 0; i < 20000; ++i) {
                int w[12];
                const int n = h.take(1 + (i + t) % 4, w);
                for (int k = 0; k < n; ++k) if (held[w[k]].fetch_add(1) != 0) twice = true;
                for (int k = 0; k < n; ++k) held[w[k]].fetch_sub(1);
                h.give(w, n);
            }
        });
    for (auto& t : threads) t.join();
    return twice.load() || h.take(12, a) != 12;
}
"""


def test_lanes_are_handed_out_without_waiting(tmp_path):
    compile_and_run(tmp_path, HANDOUT, "-pthread")
