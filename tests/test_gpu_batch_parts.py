"""GPU: steps of 33 to 64 sequences, two parts of the persistent step kernel (csrc/batch.cu) with half of the sequences and of the SMs each."""
import numpy as np
import pytest

from test_gpu_batch_edges import TILES, engine
from test_gpu_batch_failure import child
from test_gpu_batch_step import EDGES, LONG, run

pytestmark = pytest.mark.gpu


# (slots, dim, heads, ffn, vocab, layers, total, prompt lengths): one row more and one less in the second part, all rows, head sizes 64 and 128, whole and
# cut sequences; a job of fewer than 32
@pytest.mark.parametrize("slots,dim,heads,ffn,vocab,layers,total,lens", [
    (33, 320, 5, 1280, 997, 2, 512, (TILES + EDGES) * 2),
    (64, 768, 12, 3072, 1001, 2, 512, (TILES + EDGES + EDGES) * 2),
    (64, 320, 5, 1280, 997, 3, 1200, LONG * 3 + EDGES * 2 + (1000, 1024, 1100)),
    (47, 256, 2, 1184, 1000, 2, 512, TILES + EDGES * 2),
    (64, 256, 2, 1184, 997, 1, 620, LONG * 5),
    (63, 640, 5, 1280, 997, 2, 128, EDGES[:14]),
    (40, 768, 6, 3072, 997, 1, 96, EDGES + EDGES),
    (33, 1536, 12, 3072, 997, 1, 96, EDGES + EDGES),       # too wide for parts: launches
])
def test_every_sequence_is_the_oracles(ak, orc, ctx, slots, dim, heads, ffn, vocab, layers, total, lens):
    cfg = ak.ModelConfig(vocab, dim, heads, layers, total, ffn)
    params = ak.synthetic_weights(cfg, seed=slots, std=0.05)
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_BF16)
    prompts = [ak.uniform_tokens(n, vocab, seed=170 + i) for i, n in enumerate(lens)]
    new = [4 + 3 * (i % 3) for i in range(len(lens))]
    out = run(ak, ctx, w, prompts, slots, total, new, True)
    assert [o.tolist() for o in run(ak, ctx, w, prompts, slots, total, new, False)] == [o.tolist() for o in out]
    for i in (0, min(slots, len(lens)) - 1):               # sequences of the first and the last slot, alone
        assert run(ak, ctx, w, [prompts[i]], slots, total, [new[i]], True)[0].tolist() == out[i].tolist()
    om = orc.Model(cfg.as_dict(), [p if p.ndim == 1 else orc.round_bf16(p) for p in params])
    tol = 8 * np.sqrt(7 * layers + 1) * 2.0 ** -9          # as in test_gpu_batch_step
    for i, (p, o) in enumerate(zip(prompts, out)):
        s = orc.Session(om, total)
        _, logits = s.prefill(p)
        assert len(o) == min(total - len(p), new[i])
        for t in o:
            assert logits[t] >= logits.max() - tol * logits.std(), (i, len(p), o.tolist())
            _, logits = s.decode_step(int(t)) if s.cur_len < total else (0, None)
    ctx.check_device_status()
    w.close()


@pytest.mark.parametrize("dim,heads,slots,total", [(320, 5, 41, 512), (768, 12, 64, 512), (768, 12, 64, 1200), (256, 2, 64, 512), (256, 2, 40, 768)])
def test_prompts_beside_and_many_runs(ak, ctx, dim, heads, slots, total):
    """Sequences join and leave: tokens are the same in every run, with chunked prompts, and alone."""
    cfg = ak.ModelConfig(997, dim, heads, 2, total, 4 * dim if dim > 300 else 1184)
    w = ak.ModelWeights(ctx, cfg, ak.AK_BF16)
    w.init_synthetic(5, 0.05)
    prompts = [ak.uniform_tokens(1 + 29 * i % 150, 997, seed=i) for i in range(2 * slots)]
    new = [1 + 7 * i % 12 for i in range(len(prompts))]
    def job(e, which):
        ids = [e.submit(prompts[i], len(prompts[i]) + new[i]) for i in which]
        e.run_to_completion()
        out = [e.poll(i)[0].tolist() for i in ids]
        e.clear_finished()
        return out
    e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, async_steps=True)
    want = job(e, range(len(prompts)))
    for _ in range(15):
        assert job(e, range(len(prompts))) == want
    for i in range(0, len(prompts), slots // 3):
        assert job(e, [i]) == [want[i]], i
    e.close()
    e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, async_steps=True, prefill_chunk_rows=24)
    assert job(e, range(len(prompts))) == want
    e.close()
    ctx.check_device_status()
    w.close()


def test_rows_that_are_not_finite(ak, ctx):
    cfg = ak.ModelConfig(997, 320, 5, 3, 96, 1280)
    params = ak.synthetic_weights(cfg, seed=4, std=0.05)
    params[0][13] = np.nan
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_BF16)
    prompts = [15 + ak.uniform_tokens(4 + i % 20, 982, seed=i) for i in range(50)]
    clean = engine(ak, ctx, w, prompts, 50, 96, 12, False)
    for i in (1, 24, 25, 49):
        prompts[i][2] = 13
    out = engine(ak, ctx, w, prompts, 50, 96, 12, False)
    for i in range(50):
        assert out[i] == ([0] * 12 if i in (1, 24, 25, 49) else clean[i]), i
    ctx.check_device_status()
    w.close()


@pytest.mark.parametrize("async_steps", [False, True])
def test_wait_that_runs_out_in_one_part(async_steps):
    """The second part lacks a block: its waits end, and the step fails."""
    child((320, 5, 1280, 2, 40, 96, async_steps))
