"""GPU: the step of several sequences (csrc/batch.cu) at the edges of its tiles, units and buffers, every sequence of every case against the oracle;
rows that are not finite beside rows that are; many runs of one job."""
import numpy as np
import pytest

from test_gpu_batch_step import EDGES, LONG, run

pytestmark = pytest.mark.gpu
TILES = (127, 128, 129, 255, 383, 385, 480, 500)   # around the 4 and 12 tiles of 32 positions (8 and 24 of 16) that the warps of a unit have at once


# (slots, dim, heads, ffn, vocab, layers, total, prompt lengths)
@pytest.mark.parametrize("slots,dim,heads,ffn,vocab,layers,total,lens", [
    (8, 320, 5, 1280, 997, 2, 512, TILES),                              # twelve warps a unit, head size 64
    (32, 320, 5, 1280, 997, 2, 512, (TILES + EDGES) * 2),               # four warps a unit; rows 16 .. 31 in the second tile of rows
    (8, 256, 2, 1184, 997, 2, 512, TILES),                              # the same for head size 128
    (32, 640, 5, 1280, 997, 2, 512, EDGES + TILES + TILES[:8]),
    (32, 320, 5, 1280, 997, 2, 1024, LONG * 2 + (1000, 1010, 800) + EDGES[:9]),   # the longest whole sequences of head size 64
    (4, 320, 5, 1280, 997, 2, 1040, (1018, 1030, 767, 300)),            # splits from there on, with one tile of rows and with two
    (32, 320, 5, 1280, 997, 2, 1200, LONG * 2 + (1000, 1024, 1100) + EDGES[:9]),
    (32, 256, 2, 1184, 997, 2, 620, LONG * 3),                          # for head size 128 from 512 on
    (4, 320, 5, 1280, 997, 1, 96, (1, 16, 33, 60)),                     # one layer: a set is used again two steps later
    (6, 2048, 16, 8192, 997, 2, 96, (1, 16, 33, 48, 7, 12)),            # two tiles of the residual stream on an SM, K of several ring chunks
    (5, 2048, 16, 8192, 1000, 1, 700, (1, 255, 257, 600, 33)),
    (16, 3072, 24, 3072, 997, 1, 64, (1, 2, 15, 16, 17)),               # three tiles of it, six passes of qkv, the fewest ring slots
])
def test_every_sequence_is_the_oracles(ak, orc, ctx, slots, dim, heads, ffn, vocab, layers, total, lens):
    cfg = ak.ModelConfig(vocab, dim, heads, layers, total, ffn)
    params = ak.synthetic_weights(cfg, seed=slots, std=0.05)
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_BF16)
    prompts = [ak.uniform_tokens(n, vocab, seed=70 + i) for i, n in enumerate(lens)]
    new = [5 + 3 * (i % 3) for i in range(len(lens))]
    out = run(ak, ctx, w, prompts, slots, total, new, True)
    last = min(slots, len(lens)) - 1                       # the sequence of the last slot, alone
    alone = run(ak, ctx, w, [prompts[last]], slots, total, [new[last]], True)
    assert alone[0].tolist() == out[last].tolist()
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


@pytest.mark.parametrize("slots,dim,heads,ffn,layers,total", [
    (5, 320, 5, 1280, 3, 300), (20, 320, 5, 1280, 2, 1100), (4, 768, 12, 3072, 2, 300), (3, 2048, 16, 8192, 1, 200), (16, 3072, 24, 3072, 1, 200)])
def test_prompts_beside_the_step(ak, ctx, slots, dim, heads, ffn, layers, total):
    """Steps with prompts run on fewer SMs: a sequence's tokens are those it has alone, with whole prompts and with chunks."""
    cfg = ak.ModelConfig(997, dim, heads, layers, total, ffn)
    w = ak.ModelWeights(ctx, cfg, ak.AK_BF16)
    w.init_synthetic(5, 0.05)
    prompts = [ak.uniform_tokens(1 + 29 * i % 150, 997, seed=i) for i in range(3 * slots)]
    new = [1 + 7 * i % 12 for i in range(len(prompts))]
    def job(which, chunk):
        e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, async_steps=True, prefill_chunk_rows=chunk)
        ids = [e.submit(prompts[i], len(prompts[i]) + new[i]) for i in which]
        e.run_to_completion()
        out = [e.poll(i)[0].tolist() for i in ids]
        e.close()
        return out
    everything = range(len(prompts))
    out = job(everything, 0)
    assert job(everything, 0) == out and job(everything, 24) == out
    for i in list(everything)[:: max(1, slots // 3)]:
        assert job([i], 0) == [out[i]], i
    ctx.check_device_status()
    w.close()


def engine(ak, ctx, w, prompts, slots, total, new, chain):
    e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, attn_timing=chain)   # with attn_timing a step is a chain of launches
    ids = [e.submit(p, len(p) + new) for p in prompts]
    e.run_to_completion()
    out = [e.poll(i)[0].tolist() for i in ids]
    e.close()
    return out


@pytest.mark.parametrize("slots", [6, 24])
def test_rows_that_are_not_finite(ak, ctx, slots):
    """A sequence that meets a NaN picks what the launch chain picks (no logit is a maximum: token 0), and its neighbours pick what they pick without it."""
    cfg = ak.ModelConfig(997, 320, 5, 3, 96, 1280)
    params = ak.synthetic_weights(cfg, seed=4, std=0.05)
    params[0][13] = np.nan
    params[0][14, 5] = np.inf
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_BF16)
    prompts = [15 + ak.uniform_tokens(4 + i, 982, seed=i) for i in range(slots)]
    clean = engine(ak, ctx, w, prompts, slots, 96, 12, False)
    bad = {1: 13, 3: 14, slots - 1: 13}
    for i, t in bad.items():
        prompts[i][2] = t
    out = engine(ak, ctx, w, prompts, slots, 96, 12, False)
    chain = engine(ak, ctx, w, prompts, slots, 96, 12, True)
    for i in range(slots):
        assert out[i] == (chain[i] if i in bad else clean[i]), i
    assert all(out[i] == [0] * 12 for i in bad)
    ctx.check_device_status()
    w.close()


def test_sums_of_squares_that_overflow(ak, ctx):
    """1 / rms is 0 there, so every logit is 0 and the first token is picked, as by the launch chain."""
    cfg = ak.ModelConfig(997, 320, 5, 2, 96, 1280)
    params = ak.synthetic_weights(cfg, seed=4, std=0.05)
    params[0] *= np.float32(1e25)
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_BF16)
    for slots in (3, 20):
        prompts = [ak.uniform_tokens(4 + i, 997, seed=i) for i in range(slots)]
        out = engine(ak, ctx, w, prompts, slots, 96, 6, False)
        assert out == engine(ak, ctx, w, prompts, slots, 96, 6, True) and out == [[0] * 6] * slots
    ctx.check_device_status()
    w.close()


def test_many_runs_give_the_same_tokens(ak, ctx):
    for dim, heads, slots, total in ((320, 5, 21, 512), (256, 2, 8, 620), (768, 12, 32, 512), (768, 12, 32, 1200), (320, 5, 32, 1200), (320, 5, 9, 1200), (256, 2, 20, 768),
                                    (320, 5, 9, 512), (256, 2, 8, 500), (256, 2, 20, 500)):   # every form of a step of one part
        cfg = ak.ModelConfig(1000, dim, heads, 4, total, 4 * dim if dim > 300 else 1184)
        w = ak.ModelWeights(ctx, cfg, ak.AK_BF16)
        w.init_synthetic(3, 0.05)
        prompts = [ak.uniform_tokens(1 + 37 * i % 300, 1000, seed=i) for i in range(slots)]
        e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, async_steps=True)
        want = None
        for _ in range(25):
            ids = [e.submit(p, len(p) + 8 + 5 * (i % 4)) for i, p in enumerate(prompts)]
            e.run_to_completion()
            out = [e.poll(i)[0].tolist() for i in ids]
            e.clear_finished()
            assert want is None or out == want
            want = out
        e.close(); w.close()
    ctx.check_device_status()


def test_steps_are_counted_as_they_are_launched(ak, ctx):
    """A decode-only step of the persistent kernel is one launch and no graph, a step with prompts is a graph."""
    cfg = ak.ModelConfig(997, 320, 5, 2, 96, 1280)
    w = ak.ModelWeights(ctx, cfg, ak.AK_BF16)
    w.init_synthetic(3, 0.05)
    for async_steps in (False, True):
        e = ak.Engine(ctx, w, max_seqs=4, max_seq_len=96, use_cuda_graph=True, async_steps=async_steps)
        for rep in range(2):
            for i in range(4):
                e.submit(ak.uniform_tokens(5, 997, seed=i), 25)
            e.run_to_completion()
            st = e.stats()
            e.reset_stats()
            assert (st["steps"], st["graph_launches"], st["eager_steps"]) == (20, 1, 19)
        assert st["kernel_launches"] <= 19 + 30
        e.close()
    w.close()
