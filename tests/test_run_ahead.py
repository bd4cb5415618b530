"""CPU: work launched ahead of its results (csrc/ahead.h): order, the number in flight, and that nothing is under way on return."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <stdio.h>
#include "ahead.h"
// n items, `ahead` in flight; launch `bad_launch` and wait `bad_wait` fail (-1: none), wait `last` stops; the drain returns `bad_drain`
static int one(int n, int ahead, int bad_launch, int bad_wait, int last, int bad_drain) {
    int launched = 0, done = 0, flying = 0, most = 0, drains = 0;
    bool order = true;
    const int rc = ak::run_ahead(
        n, ahead,
        [&](uint32_t j) { order = order && (int)j == launched; flying++; if ((int)j == bad_launch) return 11; launched++; if (flying > most) most = flying; return 0; },
        [&](uint32_t j, bool& stop) { order = order && (int)j == done && done < launched; if ((int)j == bad_wait) return 22; flying--; done++; stop = (int)j == last; return 0; },
        [&]() { drains++; flying = 0; return bad_drain; });
    const int all = last >= 0 && last + 1 < n ? last + 1 : n;
    bool ok = order && flying == 0 && most <= ahead && drains <= 1;
    switch (rc) {
        case 0: ok = ok && done == all; break;
        case 11: ok = ok && bad_launch >= done && bad_launch < done + ahead && done < all; break;   // met while the pipe was filled
        case 22: ok = ok && done == bad_wait && done < all; break;
        case 33: ok = ok && bad_drain == 33 && drains == 1 && done == all; break;
        default: ok = false;
    }
    if (!ok) printf("n %d ahead %d launch %d wait %d last %d drain %d: rc %d done %d flying %d\n", n, ahead, bad_launch, bad_wait, last, bad_drain, rc, done, flying);
    return !ok;
}
int main() {
    int bad = 0, runs = 0;
    for (int n = 0; n <= 6; n++)
        for (int ahead = 1; ahead <= 4; ahead++)
            for (int l = -1; l < n; l++)
                for (int w = -1; w < n; w++)
                    for (int last = -1; last < n; last++)
                        for (int d = 0; d <= 33; d += 33) { bad += one(n, ahead, l, w, last, d); runs++; }
    printf("%d of %d\n", bad, runs);
    return bad != 0;
}
"""


def test_run_ahead(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    (tmp_path / "check.cpp").write_text(CHECK)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "akasha-core_b200", "csrc"), str(tmp_path / "check.cpp"), "-o", str(tmp_path / "check")], check=True)
    p = subprocess.run([str(tmp_path / "check")], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout[-2000:]
