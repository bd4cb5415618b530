"""GPU: sessions at the edges of what the batch-1 step takes, and after generation that ended early."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# A model whose ffn-down row does not fit the step kernel's ring takes the launch chain: a decode step's logits equal the last row of a
# prefill of the same tokens.
@pytest.mark.parametrize("dim,heads,ffn", [(768, 12, 20480), (320, 5, 24000)])
def test_wide_ffn_falls_back(ak, ctx, dim, heads, ffn):
    cfg = ak.ModelConfig(600, dim, heads, 1, 64, ffn)
    w = ak.ModelWeights(ctx, cfg, ak.AK_F32)
    w.init_synthetic(5, 0.02)
    s, ref = ak.InferenceSession(ctx, w, 64), ak.InferenceSession(ctx, w, 64)
    toks = ak.uniform_tokens(20, 600, seed=1)
    s.replace_cache()
    s.prefill(toks[:15])
    for j in range(15, 19):
        got, _ = s.decode_step(int(toks[j]))
        ref.replace_cache()
        want, _ = ref.prefill(toks[:j + 1])
        assert np.linalg.norm(got - want) < 2e-5 * np.linalg.norm(want)   # f32 sums of up to 24000 terms in another order
    ctx.check_device_status()
    s.close(); ref.close(); w.close()
