"""CPU: the batch-1 step's plan (csrc/solo_plan.h). Every model it accepts keeps its blocks inside the ring, its divisions exact and its
logits inside their buffer, for every SM; models that would not are refused, whatever their size."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <stdio.h>
#include <stdlib.h>
#include <initializer_list>
#include "solo_plan.h"
using namespace ak::solo;
static void fail(const char* what, uint32_t esz, uint32_t dim, uint32_t ffn, uint32_t vocab, uint32_t cta) {
    printf("FAIL %s: esz %u dim %u ffn %u vocab %u cta %u\n", what, esz, dim, ffn, vocab, cta);
    exit(1);
}
static void check(uint32_t esz, uint32_t dim, uint32_t ffn, uint32_t vocab) {
    Plan p;
    if (!make_plan(esz, dim, ffn, p) || p.smem > MAX_DYN_SMEM) fail("plan", esz, dim, ffn, vocab, 0);
    for (uint32_t cta : {0u, 1u, 73u, 147u}) {
        uint32_t n[N_KINDS] = {3 * dim, dim, ffn, dim, vocab};
        for (uint32_t i = 0; i < N_KINDS; i++) {
            Kind d;
            make_kind(d, n[i], i == 3 ? ffn : dim, esz, p.slots, cta, CTAS);
            if (d.blk == 0 || d.blk > BLK || d.blk % d.rpc) fail("block", esz, dim, ffn, vocab, cta);
            if ((uint64_t)d.rows * d.k > 0xffffffffull) fail("elements", esz, dim, ffn, vocab, cta);
            if (i == 4) {
                if ((uint64_t)d.rows * 4 > kv_bytes(esz)) fail("logits", esz, dim, ffn, vocab, cta);
                for (uint32_t j = 0; j < d.rows; j++)
                    if (div_inv(j, d.inv_rpc) != j / d.rpc) fail("row division", esz, dim, ffn, vocab, cta);
                continue;
            }
            const uint32_t per = udiv_up(d.piece, SLICE);
            for (uint32_t s = 0; s < udiv_up(d.k, SLICE); s++)
                if (d.ppr > 1 && div_inv(s, d.inv_pslices) != s / per) fail("slice division", esz, dim, ffn, vocab, cta);
            for (uint32_t j0 = 0; j0 < d.rows; j0 += d.blk) {
                const uint32_t rows = umin(d.blk, d.rows - j0), chunks = d.ppr > 1 ? rows * d.ppr : div_inv(rows + d.rpc - 1, d.inv_rpc);
                if (chunks != (d.ppr > 1 ? rows * d.ppr : udiv_up(rows, d.rpc)) || chunks > p.slots || chunks > 32) fail("chunks", esz, dim, ffn, vocab, cta);
                for (uint32_t r = 0; r < rows; r++) {
                    const uint32_t last = d.ppr > 1 ? (d.ppr - 1) * SLOT + (d.k - (d.ppr - 1) * d.piece) * esz : d.k * esz;
                    if (d.row_off[r & 3][r >> 2] + last > p.slots * SLOT) fail("ring", esz, dim, ffn, vocab, cta);
                }
            }
        }
    }
}
static uint64_t word(uint32_t value, uint32_t tag) { return (uint64_t)value | (uint64_t)tag << 32; }
static int words() {   // the host's reading of a step's done word
    uint32_t v = 7;
    if (read_word(0, 1, v) || v != 7) return 1;                        // never written
    if (read_word(word(5, 4), 8, v) || v != 7) return 2;               // an earlier step's
    if (read_word(word(STEP_FAILED, 4), 8, v) || v != 7) return 3;
    if (!read_word(word(5, 8), 8, v) || v != 5) return 4;
    if (!read_word(word(0, 0xffffffffu), 0xffffffffu, v) || v != 0) return 5;
    if (!read_word(word(STEP_FAILED, 8), 8, v) || v != STEP_FAILED) return 6;   // a wait of this step ran out: no vocabulary has that id
    return 0;
}
int main(int argc, char** argv) {
    if (argc == 2) {
        printf("%d\n", words());
        return 0;
    }
    if (argc == 7) {   // one shape: esz dim ffn heads layers vocab
        uint32_t v[6];
        for (int i = 0; i < 6; i++) v[i] = (uint32_t)strtoul(argv[i + 1], 0, 10);
        printf("%d\n", (int)shape_supported(v[0], v[1], v[2], v[3], v[4], v[5]));
        return 0;
    }
    uint32_t n = 0;
    for (uint32_t esz : {2u, 4u})
        for (uint32_t hd : {64u, 128u})
            for (uint32_t heads = 1; heads * hd * esz <= SLOT; heads++)
                for (uint32_t ffn = 148; ffn <= 32768; ffn += ffn < 512 || (ffn > 18000 && ffn < 24000) ? 4 : 124)
                    for (uint32_t vocab : {1u, 37u, 50257u, 600000u, 1000000u, 1818624u, 1818625u, 4000000u})
                        if ((vocab == 50257 || ffn == 3000 || ffn == 400) && shape_supported(esz, heads * hd, ffn, heads, 12, vocab)) {
                            check(esz, heads * hd, ffn, vocab);
                            n++;
                        }
    printf("ok %u\n", n);
    return 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("solo_plan")
    (d / "check.cpp").write_text(CHECK)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "akasha-core_b200", "csrc"), str(d / "check.cpp"), "-o", str(d / "check")], check=True)
    return lambda *a: subprocess.run([str(d / "check"), *map(str, a)], capture_output=True, text=True).stdout.strip()


def test_every_accepted_model_fits(plan):
    out = plan()
    assert out.startswith("ok") and int(out.split()[1]) > 10000, out


F32, BF16 = 4, 2


@pytest.mark.parametrize("esz,dim,ffn,heads,layers,vocab,want", [
    (F32, 768, 3072, 12, 12, 50257, 1), (BF16, 768, 3072, 12, 12, 50257, 1), (F32, 320, 1280, 5, 6, 50257, 1), (BF16, 2048, 8192, 16, 24, 50257, 1),
    (F32, 2560, 20480, 20, 2, 1000, 0),      # a ffn-down row of seven pieces, six slots
    (F32, 2560, 18432, 20, 2, 1000, 1), (F32, 2560, 18496, 20, 2, 1000, 0),
    (F32, 768, 20480, 12, 1, 1000, 0), (F32, 2048, 21504, 16, 1, 1000, 0),
    (BF16, 384, 1536, 6, 2, 606208, 1), (BF16, 384, 1536, 6, 2, 700000, 0),      # 4096 lm_head rows an SM, 16 to a chunk
    (BF16, 1536, 6144, 12, 12, 12288 * 148, 1), (BF16, 1536, 6144, 12, 12, 12288 * 148 + 1, 0),   # logits of an SM in 48 KB
])
def test_limits(plan, esz, dim, ffn, heads, layers, vocab, want):
    assert plan(esz, dim, ffn, heads, layers, vocab) == str(want)


def test_done_word(plan):
    assert plan("words") == "0"
