"""CPU: the plan of the step of several sequences (csrc/batch_plan.h). The exchange sets are used in turn by the layers and cleared in between; by what
happens before what (no timing assumed), a set is clean whenever anybody may look at it, and nobody still reads a set that is cleared."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Every warp of every SM is followed through the phases in their order, with what has certainly happened when it gets somewhere: of each SM, the clears it
# has counted itself in for, and the last phase it has published. A warp learns that from what it polls (the publisher's knowledge) and from the
# barriers inside its SM: partial sums to the epilogue, and the epilogue's arrival behind the pass before to the compute warps.
CHECK = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <vector>
#include "batch_plan.h"
using namespace ak::batch;
static uint32_t sms = SMS;   // blocks of the step
struct Known {
    int clears[SMS], phase[SMS];   // (phase: 5 * layer + 0 qkv, 1 attention, 2 out-proj, 3 ffn-up, 4 ffn-down; -1: none)
    Known() { memset(clears, 0, sizeof clears); for (uint32_t t = 0; t < sms; t++) phase[t] = -1; }
    void join(const Known& o) {
        for (uint32_t t = 0; t < sms; t++) {
            if (o.clears[t] > clears[t]) clears[t] = o.clears[t];
            if (o.phase[t] > phase[t]) phase[t] = o.phase[t];
        }
    }
};
static uint32_t dim, ffn, heads, L;
static bool counter;
static int bad;
// a look at (or a store to) the set of layer l (-1: the embedding's) with knowledge k: its last clear has happened on every SM
static void look(const Known& k, int l, const char* what, uint32_t sm) {
    const int need = l + 3 - (int)SETS;   // clears: the one at the start, then one behind each ffn-up
    if (need <= 0) return;                // that content was a launch before
    for (uint32_t t = 0; t < sms; t++)
        if (k.clears[t] < need) {
            if (!bad++) printf("layer %d %s on SM %u: SM %u has counted %d of %d clears\n", l, what, sm, t, k.clears[t], need);
            return;
        }
}
static uint32_t n_tiles(uint32_t rows, uint32_t sm) { return tile_begin(div_up(rows, 8), sm + 1, sms) - tile_begin(div_up(rows, 8), sm, sms); }
// publishers of columns [c0, c1) of a matrix's product
static Known publishers(const std::vector<Known>& pub, uint32_t rows, uint32_t c0, uint32_t c1) {
    Known k;
    for (uint32_t t = 0; t < sms; t++) {
        const uint32_t a = tile_begin(div_up(rows, 8), t, sms) * 8, b = tile_begin(div_up(rows, 8), t + 1, sms) * 8;
        if (a < c1 && c0 < b) k.join(pub[t]);
    }
    return k;
}
int main(int argc, char** argv) {
    if (argc < 7) return 2;
    dim = atoi(argv[1]); ffn = atoi(argv[2]); heads = atoi(argv[3]); L = atoi(argv[4]);
    const uint32_t rows = atoi(argv[5]), max_len = atoi(argv[6]);
    counter = argc < 9 || atoi(argv[8]);
    if (argc >= 8 && atoi(argv[7])) sms = sms_beside(dim, L, heads, rows, max_len);
    if (!shape_supported(dim, ffn, heads, L, rows, max_len)) { printf("refused\n"); return 0; }
    const Plan p = make_plan(dim, L, heads, rows, max_len);
    std::vector<std::vector<Known>> w(SMS, std::vector<Known>(NW));   // compute warps
    std::vector<Known> e(SMS), freed(SMS), x1(SMS), qkv(SMS), x2(SMS), up(SMS);
    std::vector<Known> at(rows * heads);
    for (uint32_t s = 0; s < sms; s++) { freed[s] = e[s]; e[s].clears[s] = 1; x1[s] = e[s]; }   // embedding; the clear at the start
    const uint32_t n_of[4] = {3 * dim, dim, ffn, dim}, k_of[4] = {dim, dim, dim, ffn};
    const uint32_t groups = sms * (NW / p.wpi), splits = div_up(max_len, split_len(max_len, dim / heads));
    for (uint32_t l = 0; l < L; l++)
        for (uint32_t ph = 0; ph < 4; ph++) {
            if (ph == 1) {   // attention: every unit, its warps together; one publishes
                std::vector<Known> part(rows * heads * splits);
                for (uint32_t u = 0; u < rows * heads * splits; u++) {
                    const uint32_t j = u / groups, x = u % groups, g = j & 1 ? groups - 1 - x : x, s = g % sms, w0 = g / sms * p.wpi, head = u / splits % heads;
                    Known all;
                    for (uint32_t i = w0; i < w0 + p.wpi; i++) {
                        look(w[s][i], l, "attention", s);
                        for (uint32_t m = 0; m < 3; m++) w[s][i].join(publishers(qkv, 3 * dim, m * dim + head * (dim / heads), m * dim + (head + 1) * (dim / heads)));
                        all.join(w[s][i]);
                    }
                    for (uint32_t i = w0; i < w0 + p.wpi; i++) w[s][i] = all;
                    part[u] = all;
                }
                for (uint32_t i = 0; i < rows * heads; i++) {
                    at[i] = Known();
                    for (uint32_t k = 0; k < splits; k++) at[i].join(part[i * splits + k]);
                }
            }
            std::vector<Known>& out = ph == 0 ? qkv : ph == 1 ? x2 : ph == 2 ? up : x1;
            const std::vector<Known> in = ph == 0 ? x1 : ph == 2 ? x2 : up;
            std::vector<Known> next(SMS);
            for (uint32_t s = 0; s < sms; s++) {
                const uint32_t n = n_tiles(n_of[ph], s);
                const int src = ph == 0 ? (int)l - 1 : (int)l;
                if ((ph == 0 || ph == 2) && n) {   // sums of squares
                    look(e[s], src, "norm", s);
                    e[s].join(publishers(in, dim, 0, dim));
                }
                if (ph == 1 && counter)
                    for (uint32_t t = 0; t < sms; t++)
                        if (e[s].clears[t] < (int)clears_before_out(l)) e[s].clears[t] = clears_before_out(l);
                for (uint32_t b = 0; b < n; b += TB) {
                    for (uint32_t i = 0; i < NW; i++) {
                        for (uint32_t sl = i; sl < k_of[ph] / 32; sl += NW) {
                            look(w[s][i], src, "product", s);
                            if (ph == 1) for (uint32_t r = 0; r < rows; r++) w[s][i].join(at[r * heads + sl * 32 / (dim / heads)]);
                            else w[s][i].join(publishers(in, k_of[ph], sl * 32, sl * 32 + 32));
                        }
                        w[s][i].join(freed[s]);
                        e[s].join(w[s][i]);
                    }
                    freed[s] = e[s];
                }
                next[s] = e[s];
                if (n) { look(e[s], l, "publish", s); next[s].phase[s] = 5 * l + (ph ? ph + 1 : 0); }
                if (ph == 2) {
                    // the set of layer l - 1 is cleared: who reads it (to the end: qkv of layer l) has published that phase, which is behind its reads
                    for (uint32_t t = 0; t < sms; t++) {
                        const int last = n_tiles(3 * dim, t) ? 5 * (int)l : 5 * (int)(l - 1) + (n_tiles(dim, t) ? 4 : 3);
                        if (l && t != s && e[s].phase[t] < last) {
                            if (!bad++) printf("layer %u: SM %u clears the set of layer %u, SM %u is known to be through phase %d, not %d\n", l, s, l - 1, t, e[s].phase[t], last);
                        }
                    }
                    e[s].clears[s] = l + 2;
                }
            }
            out = next;
        }
    printf(bad ? "%d bad\n" : "ok\n", bad);
    return 0;
}
"""


# A warp's walk over its cache tiles, for every length of a unit: the block table is read for the sequence's own blocks only, every tile is met
# once in its order, in every layer.
WALK = r"""
#include <stdio.h>
#include <initializer_list>
#include "batch_plan.h"
using namespace ak::batch;
int main() {
    int bad = 0, walks = 0;
    for (uint32_t up : {16u, 32u})
        for (uint32_t wpi : {4u, 6u, 12u})
            for (uint32_t place = 0; place < wpi; place++)
                for (uint32_t n0 = 1; n0 <= 512; n0 += n0 < 70 ? 1 : 61)
                    for (uint32_t n1 : {0u, 1u, 17u, 33u, 512u}) {
                        const uint32_t lens[2] = {n0, n1}, nu = n1 ? 2 : 1, L = 3;
                        auto unit_at = [&](uint32_t j) { return Unit{0, 0, 0, 0, lens[j], div_up(lens[j], up)}; };
                        Walk k{};
                        k.nu = nu;
                        k.b = place;
                        uint32_t want = 0, met = 0;
                        for (uint32_t j = nu; j-- > 0;) {
                            for (uint32_t b = place; b < unit_at(j).nb; b += wpi) want++;
                            if (place < unit_at(j).nb) { k.more = 1; k.j = j; }
                        }
                        if (!k.more) continue;
                        k.u = unit_at(k.j);
                        uint32_t last = 0;
                        auto look = [&]() {
                            if (k.b * up >= k.u.n) bad++;
                            const uint32_t at = (k.l * 2 + k.j) * 64 + k.b + 1;
                            if (at <= last || k.b % wpi != place) bad++;
                            last = at;
                            met++;
                        };
                        look();
                        while (k.more && met <= 3 * want) walk_on(k, wpi, place, L, unit_at, look);
                        if (met != 3 * want) bad++;
                        walks++;
                    }
    printf(bad ? "%d bad\n" : "ok %d\n", bad ? bad : walks);
    return 0;
}
"""


def build(tmp_path_factory, text):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("batch_plan")
    (d / "check.cpp").write_text(text)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "akasha-core_b200", "csrc"), str(d / "check.cpp"), "-o", str(d / "check")], check=True)
    return lambda *a: subprocess.run([str(d / "check"), *map(str, a)], capture_output=True, text=True).stdout.strip()


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    return build(tmp_path_factory, CHECK)


# dim 96 .. 320: SMs without rows of qkv, out-proj and ffn-down, warps without a slice of x; 768 and 2048: every SM has all kinds of rows
@pytest.mark.parametrize("dim,ffn,heads", [(128, 1184, 1), (256, 1216, 2), (320, 1280, 5), (768, 3072, 12), (1280, 2560, 10), (2048, 8192, 16)])
@pytest.mark.parametrize("rows,max_len", [(1, 512), (8, 1024), (16, 1200)])
def test_sets_are_clean_and_unread(plan, dim, ffn, heads, rows, max_len):
    for layers in (1, 2, 3, 4, 7):
        for beside in (0, 1):
            assert plan(dim, ffn, heads, layers, rows, max_len, beside) == "ok"


def test_walk_stays_in_the_block_table(tmp_path_factory):
    out = build(tmp_path_factory, WALK)()
    assert out.startswith("ok") and int(out.split()[1]) > 1000, out
