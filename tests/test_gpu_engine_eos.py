"""GPU: engines that stop at the end-of-sequence token. A run to the end launches a step before the tokens of the one before it are read, so a sequence
that ends at a token has a row in one step more, which counts for nothing; stepping by hand and runs with a limit read the tokens first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def serve(ak, ctx, w, prompts, totals, slots, drive, **kw):
    """Tokens of every sequence, steps taken and counts of an engine driven in one of four ways."""
    e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=96, **kw)
    ids = [e.submit(p, t) for p, t in zip(prompts, totals)]
    most = 1 + sum(len(p) + t + 1 for p, t in zip(prompts, totals))   # no queue takes more steps
    steps = 0
    if drive == "by hand":
        while True:
            steps += 1
            if e.step() == (0, 0):
                break
    elif drive == "by threes":
        while True:
            n = e.run_to_completion(3)
            steps += n
            if n < 3 or all(e.poll(i)[1] for i in ids):
                break
    else:
        steps = e.run_to_completion({"to the end": 1 << 30, "limit out of reach": most, "limit": most - 1}[drive])
    polled = [e.poll(i) for i in ids]
    assert all(fin for _, fin in polled)
    st = e.stats()
    e.clear_finished()
    if kw.get("stop_on_eos"):   # the blocks are back: the same queue once more
        again = [e.submit(p, t) for p, t in zip(prompts[:slots + 1], totals)]
        e.run_to_completion()
        assert [e.poll(i)[0].tolist() for i in again] == [t.tolist() for t, _ in polled[:slots + 1]]
    e.close()
    return [t.tolist() for t, _ in polled], steps, st


@pytest.mark.parametrize("dtype_name,slots,dim,heads,ffn,chunk", [
    ("f32", 3, 64, 1, 256, 0),         # launch chain
    ("bf16", 4, 64, 1, 256, 16),       # launch chain (too narrow for the persistent step), chunked prompts
    ("bf16", 5, 320, 5, 1280, 0),      # persistent step
    ("bf16", 40, 320, 5, 1280, 0),     # of two parts
    ("bf16", 40, 320, 5, 1280, 24),
])
def test_engine_stops_at_eos(ak, ctx, dtype_name, slots, dim, heads, ffn, chunk):
    V, n, new = 12, 3 * slots + 20, 14
    make = lambda eos: ak.ModelConfig(V, dim, heads, 2, 96, ffn, eos_token=eos)
    params = ak.synthetic_weights(make(V - 1), seed=slots, std=0.08)
    weights = lambda eos: ak.ModelWeights.from_params(ctx, make(eos), params, ak.AK_F32 if dtype_name == "f32" else ak.AK_BF16)
    prompts = [ak.uniform_tokens(1 + 13 * i % 60, V, seed=900 + i) for i in range(n)]
    totals = [len(p) + new for p in prompts]
    w = weights(V - 1)
    free, _, _ = serve(ak, ctx, w, prompts, totals, slots, "by hand")
    w.close()
    first = lambda out, t: out.index(t) if t in out else -1
    # the token that ends most sequences somewhere in the middle, of those that are also a first token and not in every sequence
    hits = {t: [first(o, t) for o in free] for t in range(V)}
    eos = max((t for t in range(V) if 0 in hits[t] and -1 in hits[t]), key=lambda t: sum(h > 0 for h in hits[t]))
    at = hits[eos]
    middle = [i for i in range(n) if at[i] > 0]
    assert len(middle) >= 4
    for k, i in enumerate(middle):     # it is the last token but one that length allows, the last, or neither
        totals[i] = len(prompts[i]) + min(new, at[i] + (2, 1, 9)[k % 3])
    want = [o[:t - len(p)] for o, p, t in zip(free, prompts, totals)]
    want = [o[:o.index(eos) + 1] if eos in o else o for o in want]
    pool = 6 * max(2, slots * 2 // 3)  # fewer blocks than slots could use
    w = weights(eos)
    kw = dict(stop_on_eos=True, kv_blocks=pool, prefill_chunk_rows=chunk)
    by_hand, steps, _ = serve(ak, ctx, w, prompts, totals, slots, "by hand", **kw)
    assert by_hand == want
    for drive in ("to the end", "limit out of reach", "limit", "by threes"):
        for asynchronous in (False, True):
            out, n_steps, st = serve(ak, ctx, w, prompts, totals, slots, drive, async_steps=asynchronous, **kw)
            assert out == want, drive
            assert st["decode_tokens"] == sum(len(o) for o in want) - n, drive   # (a sequence's first token is its prompt's)
            assert st["prefill_tokens"] == sum(len(p) for p in prompts)
            if drive == "limit":
                assert n_steps == steps
    ctx.check_device_status()
    w.close()
