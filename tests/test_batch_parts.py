"""CPU: a step of 33 to 64 sequences as two parts (csrc/batch_plan.h): the exchange sets of a part, on half of the SMs, and which models fit."""
import pytest

from test_batch_plan import CHECK, build

HALF = CHECK.replace("sms_beside(dim, L, heads, rows, max_len)", "atoi(argv[7]) == 1 ? SMS / 2 : sms_beside(dim, L, heads, rows, max_len, 2)")
SHAPES = r"""
#include <stdio.h>
#include <stdlib.h>
#include "batch_plan.h"
using namespace ak::batch;
int main(int argc, char** argv) {
    const uint32_t v[] = {(uint32_t)atoi(argv[1]), (uint32_t)atoi(argv[2]), (uint32_t)atoi(argv[3]), (uint32_t)atoi(argv[4]), (uint32_t)atoi(argv[5]), (uint32_t)atoi(argv[6])};
    printf("%d %u %u", shape_supported(v[0], v[1], v[2], v[3], v[4], v[5]), parts_of(v[4]), part_seqs(v[4]));
    return 0;
}
"""


@pytest.mark.parametrize("dim,ffn,heads", [(128, 1184, 1), (320, 1280, 5), (768, 3072, 12), (1280, 2560, 10), (1536, 6144, 12)])
@pytest.mark.parametrize("rows,max_len", [(17, 512), (32, 1200)])
def test_sets_of_a_part_are_clean_and_unread(tmp_path_factory, dim, ffn, heads, rows, max_len):
    plan = build(tmp_path_factory, HALF)
    for layers in (1, 2, 5):
        for sms in (1, 2):   # half of the SMs; those of a step beside prompts
            assert plan(dim, ffn, heads, layers, rows, max_len, sms) == "ok"


def test_which_shapes_are_two_parts(tmp_path_factory):
    shapes = build(tmp_path_factory, SHAPES)
    assert shapes(768, 3072, 12, 12, 32, 512) == "1 1 32"
    assert shapes(768, 3072, 12, 12, 33, 512) == "1 2 17"
    assert shapes(768, 3072, 12, 12, 64, 512) == "1 2 32"
    assert shapes(768, 3072, 12, 12, 65, 512).startswith("0")
    assert shapes(768, 3072, 6, 12, 64, 2048).startswith("1")
    assert shapes(832, 3328, 13, 12, 32, 512).startswith("1")
    for dim, heads in ((832, 13), (1024, 8), (1536, 12)):         # K of more than a chunk: launches are faster
        assert shapes(dim, 4 * dim, heads, 12, 33, 512).startswith("0")
    assert shapes(2048, 8192, 16, 24, 64, 512).startswith("0")


DEAL = r"""
#include <stdio.h>
#include <stdlib.h>
#include "batch_plan.h"
using namespace ak::batch;
int main(int argc, char** argv) {   // the rows that argv[1] slots get, longest first: parts and rows, and the largest difference of the parts' sums
    const uint32_t n = atoi(argv[1]);
    unsigned long long seen[2] = {0, 0}, sum[2] = {0, 0};
    for (uint32_t rank = 0; rank < ROWS * MAX_PARTS; rank++) {
        const uint32_t p = part_of_rank(rank), r = row_of_rank(rank);
        if (p >= MAX_PARTS || r >= ROWS || (seen[p] >> r & 1)) { printf("rank %u", rank); return 0; }
        seen[p] |= 1ull << r;
        if (rank < n && r >= part_seqs(n)) { printf("row %u", r); return 0; }
        sum[p] += rank < n ? (unsigned long long)(n - rank) * (n - rank) : 0;   // (lengths n^2, (n - 1)^2 ... 1)
    }
    const unsigned long long d = sum[0] > sum[1] ? sum[0] - sum[1] : sum[1] - sum[0];
    printf("%s", d <= (unsigned long long)n * n ? "ok" : "uneven");
    return 0;
}
"""


def test_sequences_are_dealt_evenly(tmp_path_factory):
    """Every row of both parts is written, whatever is running; the parts' positions differ by the longest sequence at most."""
    deal = build(tmp_path_factory, DEAL)
    for n in range(33, 65):
        assert deal(n) == "ok", n
