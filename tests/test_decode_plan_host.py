"""The split of a model over the decode kernel's clusters (turkce_llm_b200/csrc/decode_plan.h), on the CPU: every plan that is
accepted, over the widths, head counts, hidden sizes, cluster sizes and sequences per cluster there can be, keeps to the
tensor core's instruction shapes and inside the block's shared and tensor memory."""
from conftest import compile_and_run

CHECK = r"""
#include "decode_plan.h"
#include <cstdio>
using namespace tb;
static int failures = 0, plans = 0;
#define REQUIRE(c) do { if (!(c)) { if (++failures <= 10) printf("D %d H %d F %d C %d R %d: %s\n", D, H, F, C, R, #c); } } while (0)
int main() {
    for (int hd : {16, 32, 48, 64})
        for (int H = 1; H * hd <= 1024; ++H)
            for (int F = 16; F <= 1024; F += 16)
                for (int C = 1; C <= 16; ++C)
                    for (int R = 1; R <= 16; ++R) {
                        const int D = H * hd;
                        DcPlan p;
                        size_t smem;
                        if (!dc_plan(&p, &smem, R, D, H, F, C, R)) continue;
                        ++plans;
                        const uint32_t end = (uint32_t)smem - 1024;          // behind the alignment pad
                        REQUIRE(smem <= 227 * 1024);
                        struct { const DcProj* pr; uint32_t act; int columns; } use[4] = {
                            {&p.q, p.o_ax, 16}, {&p.o, p.o_att, 64}, {&p.g, p.o_ax, 16}, {&p.d, p.o_ah, 64}};
                        for (auto& u : use) {
                            // M = 128: 16 <= N <= 256 in steps of 16; all slices and groups of sequences; inside the accumulator
                            REQUIRE(u.pr->umma_n % 16 == 0 && u.pr->umma_n >= 16);
                            REQUIRE(u.pr->umma_n >= u.pr->slices * p.rg * 8 && u.pr->umma_n <= u.columns);
                            // the activation rows that an instruction reads
                            REQUIRE(u.act + (uint32_t)(u.pr->umma_n / 8 * u.pr->kblocks * 1024) <= end);
                            REQUIRE(u.pr->rows <= 128 && u.pr->kblocks % u.pr->chunk == 0);
                            // a 128-row read of the last tile of the ring
                            REQUIRE(p.ring_bytes + (128 - u.pr->rows) * 128 <= end);
                        }
                        REQUIRE(p.q.tiles * 16 <= DC_COL_O - DC_COL_Q && DC_COL_D + 64 <= DC_TMEM_COLS);
                        REQUIRE(p.o_bars + (2 * DC_SLOTS + 6) * 8 + 2 * DC_SLOTS * 4 + 8 <= end);
                        REQUIRE(p.P * C >= R * H && C * p.o.n >= D && C * p.g.n >= F && C * p.q.n >= 3 * D);
                        for (int i = 0; i < R * H; ++i) REQUIRE((int)((uint32_t)i * p.h_magic >> 16) == i / H);
                        for (int i = 0; i <= H; ++i) REQUIRE((int)((uint32_t)i * p.p_magic >> 16) == i / p.P);
                        for (int i = 0; i < R * (p.g.n / 8); ++i) REQUIRE((int)((uint32_t)i * p.g8_magic >> 16) == i / (p.g.n / 8));
                    }
    printf("%d plans, %d failures\n", plans, failures);
    return failures != 0 || plans < 10000;
}
"""


def test_every_plan_keeps_to_instruction_shapes_and_memory(tmp_path):
    print(compile_and_run(tmp_path, CHECK))


RULE = r"""
#include "decode_plan.h"
#include <cstdio>
using namespace tb;
int main() {
    struct { int D, H, F, S; bool cluster; } shapes[] = {
        {384, 6, 1024, 1, true}, {384, 6, 1024, 64, true}, {384, 6, 1024, 112, true}, {384, 6, 1024, 200, true}, {384, 6, 1024, 336, true},
        {384, 6, 1024, 448, false}, {384, 12, 1024, 200, true}, {384, 24, 1024, 128, false}, {64, 2, 128, 112, true}, {64, 2, 128, 256, false},
        {768, 12, 1024, 64, true}, {768, 12, 1024, 128, false}, {1024, 16, 1024, 100, true}, {1024, 16, 1024, 128, false},
        {1024, 64, 1024, 28, true}, {1024, 64, 1024, 32, false}, {1024, 64, 1024, 64, false}};
    int wrong = 0;
    for (auto& s : shapes) {
        const int fit = 7;                                   // clusters of 16 on a B200
        DcPlan p;
        size_t smem;
        bool found = false;
        for (int R = std::min(16, ceil_div(s.S, fit)); R >= 1 && !found; --R) found = dc_plan(&p, &smem, s.S, s.D, s.H, s.F, 16, R);
        if (!found || dc_pays(p, fit) != s.cluster) { printf("D %d H %d F %d S %d: R %d\n", s.D, s.H, s.F, s.S, found ? p.R : 0); ++wrong; }
    }
    return wrong;
}
"""


def test_the_cluster_kernel_is_taken_where_it_is_faster(tmp_path):
    """(the shapes that the rule was measured on)"""
    compile_and_run(tmp_path, RULE)
