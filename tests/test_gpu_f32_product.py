"""GPU: the f32 product from split operands on the tensor cores (csrc/gemm_f32_tc.cu), through prompts of f32 sessions against 64-bit arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def forward64(cfg, params, toks):
    """Keys and values of every layer and the last row's logits, in float64."""
    import torch
    P = [torch.from_numpy(np.asarray(p)).double() for p in params]
    D, H, L = cfg.dim, cfg.num_heads, cfg.num_layers
    hd, n = D // H, len(toks)
    norm = lambda x, g: x / torch.sqrt((x * x).mean(-1, keepdim=True) + cfg.norm_eps) * g
    freq = 1.0 / torch.pow(torch.tensor(10000.0), torch.arange(0, hd, 2, dtype=torch.float32) / hd)
    ang = (torch.arange(n, dtype=torch.float32)[:, None] * freq[None]).double()
    cs, sn = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    def rope(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * cs - b * sn, a * sn + b * cs), -1).reshape(x.shape)
    h = P[0][torch.from_numpy(np.asarray(toks).astype(np.int64))]
    mask = torch.ones(n, n, dtype=torch.bool).tril()
    ks, vs = [], []
    for l in range(L):
        n1, qkv, out, n2, up, down = P[1 + 6 * l:7 + 6 * l]
        q, k, v = (norm(h, n1) @ qkv).reshape(n, 3, H, hd).unbind(1)
        q, k = rope(q), rope(k)
        s = torch.einsum("ihd,jhd->hij", q, k) / np.sqrt(hd)
        p = torch.softmax(s.masked_fill(~mask, -np.inf), -1)
        h = h + torch.einsum("hij,jhd->ihd", p, v).reshape(n, D) @ out
        u = norm(h, n2) @ up
        h = h + (u * torch.sigmoid(u)) @ down
        ks.append(k.reshape(n, D).numpy())
        vs.append(v.reshape(n, D).numpy())
    return ks, vs, (norm(h[-1:], P[1 + 6 * L]) @ P[2 + 6 * L])[0].numpy()


# K of several blocks, not a multiple of a block (64) nor of a half (32); two segments to six, in groups of one to three; columns that end inside
# a tile; rows at the edges of the 128-row tile and of the eight rows a warp splits. 64: (n, k) that stay on the FMA pipe; 65 and 101: K that is no multiple of 4
@pytest.mark.parametrize("dim,heads,ffn,vocab", [(64, 1, 100, 33), (132, 3, 260, 129), (320, 5, 1280, 997), (768, 12, 3072, 1000), (1088, 17, 36, 64),
                                                 (64, 1, 65, 33), (320, 5, 1281, 129), (384, 6, 700, 513), (256, 4, 1540, 1000)])
def test_prompt_against_64_bits(ak, ctx, dim, heads, ffn, vocab):
    cfg = ak.ModelConfig(vocab, dim, heads, 2, 600, ffn)
    params = ak.synthetic_weights(cfg, seed=dim, std=0.05)
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_F32)
    s = ak.InferenceSession(ctx, w, 600)
    for n in (1, 2, 9, 63, 127, 128, 129, 300, 520):
        toks = ak.uniform_tokens(n, vocab, seed=n)
        ks, vs, want = forward64(cfg, params, toks)
        s.replace_cache()
        logits, _ = s.prefill(toks)
        # Sums of up to 3072 terms, each rounded to 2^-24 of a partial sum a few dozen times: 2e-7 in the norm; about ten such products one behind another
        err = lambda a, b: np.linalg.norm(np.asarray(a, np.float64).ravel() - b.ravel()) / np.linalg.norm(b)
        for l in range(2):
            k, v = s.read_cache(l)
            assert err(k, ks[l]) < 2e-6 and err(v, vs[l]) < 2e-6, (n, l)
        assert err(logits, want) < 2e-6, n
    ctx.check_device_status()
    s.close(); w.close()


@pytest.mark.parametrize("dim,heads,ffn", [(64, 1, 256), (128, 2, 512), (320, 5, 1280), (384, 6, 1536), (768, 12, 3072)])
def test_rows_do_not_depend_on_their_number(ak, ctx, dim, heads, ffn):
    """Bits: whoever adds the segments of K (a CTA, a cluster of two, a CTA each), and on either pipe."""
    cfg = ak.ModelConfig(97, dim, heads, 2, 600, ffn)
    w = ak.ModelWeights.from_params(ctx, cfg, ak.synthetic_weights(cfg, seed=dim, std=0.05), ak.AK_F32)
    s = ak.InferenceSession(ctx, w, 600)
    toks = ak.uniform_tokens(600, 97, seed=1)
    def prefix(n):
        s.replace_cache()
        s.prefill(toks[:n])
        return [np.asarray(x).reshape(n, -1).copy() for x in s.read_cache(0)]
    full = prefix(600)
    for n in (1, 2, 9, 40, 64, 65, 128, 129, 300, 385, 520):
        for a, b in zip(prefix(n), full):
            assert np.array_equal(a, b[:n]), n
    ctx.check_device_status()
    s.close(); w.close()


def test_rows_that_are_not_finite(ak, ctx):
    """Rows before an infinite one are what they are without it; the row itself is not finite (its norm has no value)."""
    cfg = ak.ModelConfig(50, 320, 5, 1, 200, 1280)
    params = ak.synthetic_weights(cfg, seed=2, std=0.05)
    params[0][7, 3] = np.inf
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_F32)
    s = ak.InferenceSession(ctx, w, 200)
    toks = 8 + ak.uniform_tokens(150, 42, seed=1)
    s.replace_cache(); s.prefill(toks)
    clean = s.read_cache(0)
    toks[130] = 7
    s.replace_cache(); s.prefill(toks)
    for a, b in zip(clean, s.read_cache(0)):
        a, b = np.asarray(a).reshape(150, -1), np.asarray(b).reshape(150, -1)
        rows = np.arange(150) != 130
        assert np.array_equal(a[rows], b[rows]) and not np.isfinite(b[130]).any()
    ctx.check_device_status()
    s.close(); w.close()


def test_results_that_are_not_finite_or_nearly_so(ak, ctx):
    """Values of layer 0 (products alone, no rotation): a weight that rounds to an infinity in 16 bits but whose products are finite, an infinite one, a NaN."""
    cfg = ak.ModelConfig(50, 320, 5, 1, 300, 1280)
    params = ak.synthetic_weights(cfg, seed=3, std=0.05)
    params[1][17] = 0.05                            # (the factor of the largest weight stays below 1)
    value = params[2][:, 2 * cfg.dim:]
    value[:, 5] = 0
    value[17, 5] = 3.4e38
    value[23, 9] = -np.inf
    value[300, 130] = np.nan
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_F32)
    s = ak.InferenceSession(ctx, w, 300)
    for n in (2, 9, 130, 300):
        toks = ak.uniform_tokens(n, 50, seed=n)
        want = forward64(cfg, params, toks)[1][0]
        s.replace_cache()
        s.prefill(toks)
        got = np.asarray(s.read_cache(0)[1], np.float64).reshape(n, -1)
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(got[:, 130]).all()
        assert np.array_equal(got[:, 9], want[:, 9]) and np.isinf(got[:, 9]).all()
        for cols in ([5], [c for c in range(cfg.dim) if c not in (5, 9, 130)]):
            assert np.isfinite(got[:, cols]).all()
            assert np.linalg.norm(got[:, cols] - want[:, cols]) < 1e-6 * np.linalg.norm(want[:, cols])   # (one product, as above)
    ctx.check_device_status()
    s.close(); w.close()


@pytest.mark.parametrize("case", ["one sign", "2^-112", "2^-118"])
def test_operands_of_one_sign_and_tiny_ones(ak, ctx, case):
    """Values of layer 0 against 64 bits. Of one sign: the cut additions of the tensor cores all err the same way. Tiny weights: their third piece is lost, up
    to half of bf16's smallest number (2^-134), in 768 roundings of either sign."""
    cfg = ak.ModelConfig(50, 768, 12, 1, 200, 3072)
    params = ak.synthetic_weights(cfg, seed=3, std=0.05)
    value = params[2][:, 2 * cfg.dim:]
    if case == "one sign":
        params[0][:] = np.abs(params[0])
        value[:] = np.abs(value)
        bound = 4e-7       # 64 products: 16 of an MMA cut to 2^-24 of the largest sum each time, 4 MMAs; 0.85e-7 measured
    else:
        e = int(case[2:])
        value[:] = np.sign(value) * np.float32(2.0) ** e * (1 + np.abs(value))
        bound = 4e-7 + 2.0 ** (-134 - e)
    w = ak.ModelWeights.from_params(ctx, cfg, params, ak.AK_F32)
    s = ak.InferenceSession(ctx, w, 200)
    for n in (3, 150):
        toks = ak.uniform_tokens(n, 50, seed=n)
        want = forward64(cfg, params, toks)[1][0]
        s.replace_cache()
        s.prefill(toks)
        got = np.asarray(s.read_cache(0)[1], np.float64).reshape(n, -1)
        err = np.linalg.norm(got - want) / np.linalg.norm(want)
        print(case, n, err)
        assert err < bound
    ctx.check_device_status()
    s.close(); w.close()
