"""GPU: the step of several sequences (csrc/batch.cu) where its waits run out. The launch is a block short, so that what the others wait for never comes;
every wait has the step's time limit. In processes of their own: the device status words stay set."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys, time
sys.path.insert(0, %(root)r)
import __graft_entry__ as entry
ak = entry.load_package()
dim, heads, ffn, layers, slots, total, async_steps = %(shape)r
cfg = ak.ModelConfig(997, dim, heads, layers, total, ffn)
ctx = ak.Context(0)
w = ak.ModelWeights(ctx, cfg, ak.AK_BF16)
w.init_synthetic(1, 0.05)
make = lambda: ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, use_cuda_graph=True, async_steps=async_steps)
prompts = [ak.uniform_tokens(3 + 5 * i %% 70, 997, seed=i) for i in range(slots)]
def fill(e):
    return [e.submit(p, min(total, len(p) + 9)) for p in prompts]
good = make()
ids = fill(good)
good.run_to_completion()
want = [good.poll(i)[0].tolist() for i in ids]
e = make()
ids = fill(e)
e.step(); e.step()
e.drill_wait(4000000)   # 2 ms
codes, t0 = [], time.perf_counter()
for _ in range(4):
    try:
        e.step()
        codes.append(0)
    except ak.AkashaError as x:
        codes.append(x.code)
print("codes", codes, "seconds", time.perf_counter() - t0)
first = codes.index(104)
assert first <= (1 if async_steps else 0), codes
%(more)s
e.close()
# the device is as usable as before
ids = fill(good)
good.run_to_completion()
assert [good.poll(i)[0].tolist() for i in ids] == want
good.close(); w.close(); ctx.close()
assert time.perf_counter() - t0 < 20
print("CHILD OK")
"""


def child(shape, more=""):
    p = subprocess.run([sys.executable, "-c", CHILD % {"root": ROOT, "shape": shape, "more": more}], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert p.returncode == 0 and "CHILD OK" in p.stdout, (p.stdout[-1500:], p.stderr[-3000:])


# one and two tiles of rows, with and without splits, SMs with all and with few kinds of rows
SHAPES = [(320, 5, 1280, 2, 3, 96, True), (256, 2, 1184, 3, 20, 700, False), (768, 12, 3072, 2, 8, 512, True), (512, 4, 2048, 2, 32, 96, False), (320, 5, 1280, 2, 20, 1100, True)]


def test_the_engine_takes_no_further_step():
    """Every later call reports the error without launching anything, and so does the device status, which knows the kernel."""
    for shape in SHAPES[:2]:
        child(shape, """
assert all(c == 104 for c in codes[first:]), codes
for call in (e.step, e.run_to_completion, lambda: e.poll(ids[0]), ctx.check_device_status):
    n0 = ak.lib().ak_launch_count()
    try:
        call()
        raise SystemExit("no error")
    except ak.AkashaError as x:
        assert x.code == 104 and ak.lib().ak_launch_count() == n0, x
""")


@pytest.mark.parametrize("shape", SHAPES)
def test_a_wait_that_runs_out_is_an_error(shape):
    child(shape)
