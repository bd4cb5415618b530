"""GPU: the decode step of up to 32 sequences as one persistent kernel (csrc/batch.cu), through the engine. The oracle (f32 arithmetic on the
same bf16 weights) is fed the engine's tokens: every one of them has to be the oracle's choice but for rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def step_by_step(e):
    """The queue to its end, every step's tokens read before the next is launched (a run to the end launches ahead of them, whatever async_steps says)."""
    n = 1
    while e.step() != (0, 0):
        n += 1
    return n


def run(ak, ctx, w, prompts, slots, total, new, async_steps):
    e = ak.Engine(ctx, w, max_seqs=slots, max_seq_len=total, use_cuda_graph=True, async_steps=async_steps)
    ids = [e.submit(p, min(total, len(p) + n)) for p, n in zip(prompts, new)]
    e.run_to_completion() if async_steps else step_by_step(e)
    out = [e.poll(i)[0] for i in ids]
    e.close()
    return out


# slots on both sides of the 8 and 16 rows of the products' tiles; contexts around the 16 positions of a pool block, the 16 or 32 of an attention tile
# and the 256 of a unit of long sequences; a vocabulary that is no multiple of 8, K that is no multiple of a ring chunk, head sizes 64 and 128
EDGES = (1, 2, 7, 14, 15, 16, 17, 30, 31, 32, 33, 47, 48, 63, 64, 65)
LONG = (3, 244, 250, 255, 256, 257, 500, 511, 512, 600)


@pytest.mark.parametrize("slots,dim,heads,ffn,vocab,layers,total,lens", [
    (1, 320, 5, 1280, 997, 2, 96, (1, 30)),
    (8, 320, 5, 1280, 1000, 3, 512, EDGES),
    (9, 256, 2, 1184, 997, 2, 128, EDGES),
    (16, 768, 12, 3072, 1001, 2, 512, EDGES),
    (17, 320, 5, 1280, 997, 2, 96, EDGES + EDGES),
    (32, 256, 2, 1216, 1000, 4, 96, EDGES + EDGES + EDGES[:5]),
    (5, 320, 5, 1280, 997, 2, 700, LONG),
    (20, 256, 2, 1184, 1000, 2, 620, LONG + LONG),
])
def test_tokens_are_the_oracles(ak, orc, ctx, slots, dim, heads, ffn, vocab, layers, total, lens):
    cfg = ak.ModelConfig(vocab, dim, heads, layers, total, ffn)
    params = ak.synthetic_weights(cfg, seed=slots, std=0.05)
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_BF16)
    prompts = [ak.uniform_tokens(n, vocab, seed=10 + i) for i, n in enumerate(lens)]
    new = [6 + 5 * (i % 3) for i in range(len(lens))]      # sequences leave and join while others go on
    out = run(ak, ctx, w, prompts, slots, total, new, True)
    again = run(ak, ctx, w, prompts, slots, total, new, False)
    assert [o.tolist() for o in out] == [o.tolist() for o in again]
    alone = run(ak, ctx, w, [prompts[-1]], slots, total, [new[-1]], True)
    assert alone[0].tolist() == out[-1].tolist()
    om = orc.Model(cfg.as_dict(), [p if p.ndim == 1 else orc.round_bf16(p) for p in params])
    # 7 roundings to bf16 (2^-9 of the value at most) per layer and one before the lm_head, each as if it were an error of the logits; two logits
    # compared, four standard deviations each
    tol = 8 * np.sqrt(7 * layers + 1) * 2.0 ** -9
    for p, o in list(zip(prompts, out))[:12]:
        s = orc.Session(om, total)
        _, logits = s.prefill(p)
        for t in o:
            assert logits[t] >= logits.max() - tol * logits.std(), (len(p), o.tolist())
            _, logits = s.decode_step(int(t)) if s.cur_len < total else (0, None)
    ctx.check_device_status()
    w.close()
