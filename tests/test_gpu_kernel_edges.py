"""GPU: the kernels at the edges of their dispatch rules and tiles (remainders, the smallest and largest sizes of a variant),
against plain float64 / float32 references of the same operation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def host(t):
    return t.float().cpu().numpy()


# the streaming RMSNorm (more than 2048 rows): every register width, a row count that leaves a short last CTA
@pytest.mark.parametrize("rows,size,hd,with_res", [(2049, 320, 64, True), (2053, 320, 0, False), (2500, 384, 0, True), (2051, 768, 64, False),
                                                   (4097, 1024, 128, True), (2050, 2048, 128, False), (2049, 2048, 32, True), (9001, 196, 4, False)])
@pytest.mark.parametrize("out_dtype", [0, 1])
def test_rmsnorm_stream(ak, torch_cuda, rows, size, hd, with_res, out_dtype):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows + size)
    x = torch.randn(rows, size, device="cuda", generator=g)
    r = torch.randn(rows, size, device="cuda", generator=g) if with_res else None
    w = 1.0 + 0.1 * torch.randn(size, device="cuda", generator=g)
    pos = torch.randint(0, 4096, (rows,), device="cuda", generator=g, dtype=torch.int32)
    h = x + r if with_res else x.clone()
    want = (h.double() * torch.rsqrt(h.double().square().mean(-1, keepdim=True) + 1e-5) * w.double())
    if hd:
        # the angle is formed in f32 (position times a f32 frequency), as the reference forms it
        freq = 1.0 / torch.pow(torch.tensor(10000.0), torch.arange(0, hd, 2, dtype=torch.float32) / hd).cuda()
        ang = (pos.float()[:, None] * freq[None, :]).double().repeat(1, size // hd)
        a, b = want[:, 0::2].clone(), want[:, 1::2].clone()
        want[:, 0::2], want[:, 1::2] = a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()
    y = torch.full((rows, size), float("nan"), device="cuda", dtype=torch.float32 if out_dtype == 0 else torch.bfloat16)
    ak.ops.rmsnorm_rope_residual(x, r, w, y, pos if hd else None, rows, size, 1e-5, hd, out_dtype)
    torch.cuda.synchronize()
    # f32: a frequency one ulp off turns position 4095 by 4095 * 2^-24 ~ 2.5e-4 rad on values up to ~5; bf16: half an ulp of 2^-8
    tol = 2e-3 if out_dtype == 0 else 2e-3 + 5.0 * 2.0 ** -8
    assert float((y.double() - want).abs().max()) < tol
    if with_res:
        assert torch.equal(x, h)


# the CTA-pair GEMM's two output paths: TMA pieces (tails in m and n, a padded pitch) and direct stores (pitch no multiple of 16 bytes)
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
@pytest.mark.parametrize("m,n,k,ldc", [(1024, 256, 64, 256), (1025, 300, 136, 304), (1311, 391, 72, 392), (1311, 391, 72, 391), (2049, 257, 320, 259),
                                       (1281, 1000, 8, 1000)])
def test_gemm_pair_outputs(ak, torch_cuda, epi, m, n, k, ldc):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    wt = (0.25 * torch.randn(n, k, device="cuda", generator=g)).bfloat16()
    cdt = torch.float32 if epi <= 1 else torch.bfloat16
    c = torch.full((m, ldc), 3.0, device="cuda", dtype=cdt)
    ak.ops.gemm_bf16(a, wt, c, m, n, k, epi, ldc=ldc)
    torch.cuda.synchronize()
    acc = a.double() @ wt.double().T
    want = {0: acc, 1: acc + 3.0, 2: acc, 3: acc / (1.0 + (-acc).exp())}[epi]
    scale = float(acc.abs().max())
    # f32: k sums in f32; bf16: half an ulp of the largest value
    tol = 2.0 ** -22 * k * max(1.0, scale) + 1e-6 if epi <= 1 else 2.0 ** -8 * max(1.0, scale)
    assert float((c[:, :n].double() - want).abs().max()) < tol
    assert bool((c[:, n:] == 3.0).all())
    ak.check(ak.lib().ak_check_device_status(None))


# The batch-1 step kernel: a decode step's logits equal the last row of a prefill of the same tokens (another set of kernels).
# Shapes: one slice of K per warp or none; fewer rows than SMs; rows in pieces (ffn wider than a ring slot) and several row
# blocks per SM; head_dim 128; positions that need 1, 2, 3, 4 splits and several rounds of cache tiles, at block boundaries.
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("vocab,dim,heads,layers,ffn,lens", [
    (37, 64, 1, 2, 256, (1, 15, 16, 17)),
    (1000, 320, 5, 2, 1280, (1, 33, 191, 192, 300)),
    (50257, 768, 12, 1, 3072, (95, 96, 97, 383, 385, 700)),
    (777, 1024, 8, 2, 6200, (8, 127, 129, 640)),
    (601, 2048, 16, 1, 8192, (40, 257)),
])
def test_solo_step_equals_prefill(ak, ctx, dtype, vocab, dim, heads, layers, ffn, lens):
    cfg = ak.ModelConfig(vocab, dim, heads, layers, 1024, ffn)
    w = ak.ModelWeights(ctx, cfg, dtype)
    w.init_synthetic(5, 0.05)
    s, ref = ak.InferenceSession(ctx, w, 768), ak.InferenceSession(ctx, w, 768)
    for n in lens:
        toks = ak.uniform_tokens(n + 3, vocab, seed=n)
        s.replace_cache()
        s.prefill(toks[:n])
        for j in range(3):
            got, am = s.decode_step(int(toks[n + j]))
            ref.replace_cache()
            want, _ = ref.prefill(toks[:n + j + 1])
            assert np.isfinite(got).all() and am == int(np.argmax(got))
            rel = np.linalg.norm(got.astype(np.float64) - want) / np.linalg.norm(want.astype(np.float64))
            # f32: sums of up to 8192 terms in another order; bf16: the prefill rounds its activations to bf16 (2^-9 each, a dozen per layer)
            assert rel < (2e-5 if dtype == 0 else 2e-2), (n, j, rel)
    ctx.check_device_status()
    s.close(); ref.close(); w.close()


# the candidate list of the sampler: a small vocabulary, ties that overflow the list, k close to the thread count
@pytest.mark.parametrize("n,k,kind", [(40, 40 - 1, "random"), (300, 7, "random"), (50257, 40, "ties"), (50257, 1000, "random"), (5000, 1024, "few"), (50257, 40, "zeros")])
def test_sampler_candidates(ak, orc, torch_cuda, n, k, kind):
    torch = torch_cuda
    rng = np.random.default_rng(n + k)
    logits = (rng.standard_normal((3, n)) * 2.0).astype(np.float32)
    if kind == "ties":
        logits = np.round(logits)                 # thousands of equal logits: index order decides
    if kind == "zeros":
        logits[:] = np.where(rng.random((3, n)) < 0.5, -0.0, 0.0)
    if kind == "few":
        logits[:, 50:] = -1e30
    d = torch.from_numpy(logits).cuda()
    for step in range(6):
        out = torch.full((3,), -1, dtype=torch.int32, device="cuda")
        ak.ops.sample_token(d, 3, n, out, 1.3, k, 0.97, 99, step)
        got = out.cpu().numpy()
        for r in range(3):
            assert int(got[r]) == orc.sample_token(logits[r], 1.3, k, 0.97, np.zeros(0, np.uint32), 1.0, r=ak.ops.sampler_uniform(99, step, r))


# Prefill attention with more items than SMs (two query tiles per block, the persistent path): tile and block edges, an empty
# sequence, scores that grow by more than the rescaling threshold. A sequence alone (one query tile per block, its own launch)
# gives the same bits.
@pytest.mark.parametrize("heads,hd", [(12, 64), (16, 128)])
@pytest.mark.parametrize("q_scale", [1.0, 12.0])
def test_attn_prefill_many_items(ak, torch_cuda, heads, hd, q_scale):
    torch = torch_cuda
    lens = [257, 1, 128, 0, 129, 255, 256, 127, 384, 385, 511, 513, 640, 17, 700]
    g = torch.Generator(device="cuda").manual_seed(hd)
    n, mx = len(lens), max(lens)
    mb = (mx + 15) // 16
    nb = n * mb
    kp, vp = (torch.randn(nb, heads, 16, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    tables = torch.randperm(nb, device="cuda", generator=g).to(torch.int32).reshape(n, mb)
    for i, L in enumerate(lens):                      # what was never written may hold anything
        for b in range(mb):
            used = min(max(L - b * 16, 0), 16)
            if used < 16:
                vp[tables[i, b].long(), :, used:] = float("nan") if used else vp[tables[i, b].long(), :, used:]
    cu = np.zeros(n + 1, np.int32)
    cu[1:] = np.cumsum(lens)
    rows = int(cu[-1])
    q = (torch.randn(rows, heads * hd, device="cuda", generator=g) * q_scale).bfloat16()
    slot = torch.arange(n, dtype=torch.int32, device="cuda")
    run = lambda qq, tt, c, out, k, m: ak.ops.attn_prefill_paged(qq, kp, vp, tt, mb, torch.from_numpy(c).cuda(), slot, out, k, m, qq.shape[0], heads, hd,
                                                                 hd ** -0.5, ak.AK_BF16, nb)
    out = torch.full_like(q, float("nan"))
    run(q, tables, cu, out, n, mx)
    ak.check(ak.lib().ak_check_device_status(None))
    for i, L in enumerate(lens):
        if not L:
            continue
        rows_i = slice(int(cu[i]), int(cu[i + 1]))
        k, v = (p[tables[i].long()].transpose(1, 2).reshape(mb * 16, heads, hd)[:L].double().transpose(0, 1) for p in (kp, vp))
        s = torch.einsum("lhd,hkd->hlk", q[rows_i].double().reshape(L, heads, hd), k) * hd ** -0.5
        s.masked_fill_(torch.ones(L, L, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
        want = torch.einsum("hlk,hkd->lhd", s.softmax(-1), v).reshape(L, -1)
        # P is rounded to bf16 on both sides of the quotient (2 * 2^-9 of the largest value), the output once more
        tol = (2 ** -8 + 2 ** -9) * float(v.abs().max())
        assert float((out[rows_i].double() - want).abs().max()) < tol, (i, L)
        alone = torch.empty_like(q[rows_i])
        run(q[rows_i].contiguous(), tables[i:i + 1].contiguous(), np.array([0, L], np.int32), alone, 1, L)
        assert torch.equal(alone, out[rows_i]), (i, L)
    ak.check(ak.lib().ak_check_device_status(None))


# Prompts of 1024 rows and more (the CTA-pair kernel, its K segmented as the skinny launches split it) give the tokens that they
# give when they are prefilled in chunks beside a decoding sequence (skinny launches): the row's sums have the same bits.
@pytest.mark.parametrize("dim,heads,ffn", [(320, 5, 1280), (768, 12, 3072), (2048, 16, 8192)])
def test_gemm_pair_segments(ak, ctx, dim, heads, ffn):
    cfg = ak.ModelConfig(1000, dim, heads, 2, 2048, ffn)
    w = ak.ModelWeights(ctx, cfg, ak.AK_BF16)
    w.init_synthetic(7, 0.05)
    prompts = [ak.uniform_tokens(n, 1000, seed=n) for n in (3, 1024, 1290)]
    out = []
    for chunk in (0, 100):
        e = ak.Engine(ctx, w, max_seqs=3, max_seq_len=1400, prefill_chunk_rows=chunk)
        ids = [e.submit(prompts[0], 1400)]
        e.step()
        ids += [e.submit(p, p.size + 40) for p in prompts[1:]]
        e.run_to_completion()
        out.append([e.poll(i)[0].tolist()[:200] for i in ids])
        e.close()
    assert out[0] == out[1]
    ctx.check_device_status()
    w.close()


# a few long rows: a block per row (up to 148 rows), the warp-per-row kernel above; the same bits on both sides
@pytest.mark.parametrize("size", [1028, 1536, 2048, 4096])
def test_rmsnorm_wide(ak, torch_cuda, size):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(size)
    x = torch.randn(149, size, device="cuda", generator=g)
    w = 1.0 + 0.1 * torch.randn(size, device="cuda", generator=g)
    y = [torch.empty(149, size, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    ak.ops.rmsnorm_rope_residual(x, None, w, y[0], None, 149, size, 1e-5, 0, ak.AK_BF16)
    for r0, n in ((0, 1), (1, 148)):
        ak.ops.rmsnorm_rope_residual(x[r0:], None, w, y[1][r0:], None, n, size, 1e-5, 0, ak.AK_BF16)
    assert torch.equal(y[0], y[1])
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    assert float(((y[1].double() - want).abs() / (want.abs() + 1e-6)).max()) < 2 ** -8   # one rounding to bf16


# The automatic division of a sequence: whole up to 256 positions (640 where counters have to be cleared), else, with few
# sequences, in pieces of at least 4 blocks.
@pytest.mark.parametrize("rows,heads,hd,dtype,lens", [
    (1, 12, 64, 1, (1, 255, 256, 257, 639, 640, 641, 900)),
    (3, 5, 64, 0, (256, 257, 700)),
    (2, 16, 128, 1, (1, 1024, 1025, 2100)),
])
def test_attn_decode_auto_splits(ak, torch_cuda, rows, heads, hd, dtype, lens):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows)
    mx = max(lens)
    mb = (mx + 15) // 16
    tdt = torch.bfloat16 if dtype else torch.float32
    kp, vp = (torch.randn(rows * mb, heads, 16, hd, device="cuda", generator=g).to(tdt) for _ in range(2))
    tables = torch.randperm(rows * mb, device="cuda", generator=g).to(torch.int32).reshape(rows, mb)
    q = torch.randn(rows, heads * hd, device="cuda", generator=g).to(tdt)
    for step in range(len(lens) if rows == 1 else 1):
        kv = [lens[(r + step) % len(lens)] for r in range(rows)]
        out = torch.empty_like(q)
        scratch = torch.full((ak.ops.attn_decode_scratch_bytes(rows, heads, hd, mb, 0, dtype) + 16,), 255, device="cuda", dtype=torch.uint8)
        ak.ops.attn_decode_paged(q, kp, vp, tables, torch.tensor(kv, dtype=torch.int32, device="cuda"), out, rows, heads, hd, mb, hd ** -0.5, dtype, 0,
                                 rows * mb, scratch)
        ak.check(ak.lib().ak_check_device_status(None))
        for r in range(min(rows, 8)):
            k, v = (p[tables[r].long()].transpose(1, 2).reshape(mb * 16, heads, hd)[:kv[r]].double().transpose(0, 1) for p in (kp, vp))
            s = torch.einsum("hd,hkd->hk", q[r].double().reshape(heads, hd), k) * hd ** -0.5
            want = torch.einsum("hk,hkd->hd", s.softmax(-1), v).reshape(-1)
            # bf16: P rounded on both sides of the quotient, the output once; f32: sums of a few hundred terms
            tol = ((2 ** -8 + 2 ** -9) if dtype else 1e-5) * float(v.abs().max())
            assert float((out[r].double() - want).abs().max()) < tol, (r, kv[r])


# f32 prefill attention around the lines between 16-, 32- and 64-row query tiles, with lengths at the edges of a tile
@pytest.mark.parametrize("heads,hd,lens", [(12, 64, (192,)), (12, 64, (193,)), (12, 64, (512, 31)), (12, 64, (65, 577, 1, 33, 640)), (5, 128, (512, 513))])
def test_attn_prefill_f32_tiles(ak, torch_cuda, heads, hd, lens):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    n, mx = len(lens), max(lens)
    mb = (mx + 15) // 16
    kp, vp = (torch.randn(n * mb, heads, 16, hd, device="cuda", generator=g) for _ in range(2))
    tables = torch.randperm(n * mb, device="cuda", generator=g).to(torch.int32).reshape(n, mb)
    cu = np.zeros(n + 1, np.int32)
    cu[1:] = np.cumsum(lens)
    q = torch.randn(int(cu[-1]), heads * hd, device="cuda", generator=g)
    out = torch.full_like(q, float("nan"))
    ak.ops.attn_prefill_paged(q, kp, vp, tables, mb, torch.from_numpy(cu).cuda(), torch.arange(n, dtype=torch.int32, device="cuda"), out, n, mx, int(cu[-1]),
                              heads, hd, hd ** -0.5, ak.AK_F32, n * mb)
    for i, L in enumerate(lens):
        r = slice(int(cu[i]), int(cu[i + 1]))
        k, v = (p[tables[i].long()].transpose(1, 2).reshape(mb * 16, heads, hd)[:L].double().transpose(0, 1) for p in (kp, vp))
        s = torch.einsum("lhd,hkd->hlk", q[r].double().reshape(L, heads, hd), k) * hd ** -0.5
        s.masked_fill_(torch.ones(L, L, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
        want = torch.einsum("hlk,hkd->lhd", s.softmax(-1), v).reshape(L, -1)
        assert float((out[r].double() - want).abs().max()) < 2e-5, (i, L)   # f32 sums of up to 640 terms


# The activation box of a skinny GEMM: 16, 32, 64, then exactly the rows (slots of whole swizzle atoms), then 128
@pytest.mark.parametrize("m", [1, 8, 16, 17, 33, 48, 49, 64, 65, 71, 72, 73, 100, 127, 128, 129])
@pytest.mark.parametrize("n,k", [(2304, 768), (768, 3072)])
def test_gemm_skinny_rows(ak, torch_cuda, m, n, k):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, w = (torch.randn(r, k, device="cuda", generator=g).bfloat16() for r in (m, n))
    c = torch.full((m + 1, n), 3.0, device="cuda")
    ak.ops.gemm_bf16(a, w, c, m, n, k, ak.EPI_STORE_F32)
    want = a.double() @ w.double().T
    # exact products, k f32 additions of rounding 2^-24 each on partial sums of about sqrt(k): k^0.5 * k^0.5 * 2^-24, x8 for the extremes
    assert float((c[:m].double() - want).abs().max()) < 8 * k * 2.0 ** -24
    assert bool((c[m] == 3.0).all())
    ak.check(ak.lib().ak_check_device_status(None))


# f32 prefill attention: 16-, 32- and 64-row query tiles, the choice going by the CTAs of the launch. A prompt alone (each tile in turn) and
# with enough others for the largest tile: the same bits. The line between two tiles: 12 heads x 12 tiles are 144 CTAs, x 13 are 156.
@pytest.mark.parametrize("heads,hd,L", [(12, 64, 192), (12, 64, 193), (12, 64, 384), (12, 64, 385), (5, 64, 464), (5, 64, 465), (16, 128, 144), (16, 128, 145), (16, 128, 289)])
def test_attn_prefill_f32_tile_choice(ak, torch_cuda, heads, hd, L):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(L)
    n, mb = 8, (L + 15) // 16
    kp, vp = (torch.randn(n * mb, heads, 16, hd, device="cuda", generator=g) for _ in range(2))
    tables = torch.randperm(n * mb, device="cuda", generator=g).to(torch.int32).reshape(n, mb)
    q = torch.randn(n * L, heads * hd, device="cuda", generator=g)
    outs = []
    for k in (1, n):
        cu = torch.arange(0, (k + 1) * L, L, dtype=torch.int32, device="cuda")
        out = torch.full((k * L, heads * hd), float("nan"), device="cuda")
        ak.ops.attn_prefill_paged(q[:k * L].contiguous(), kp, vp, tables, mb, cu, torch.arange(k, dtype=torch.int32, device="cuda"), out, k, L, k * L, heads, hd,
                                  hd ** -0.5, ak.AK_F32, n * mb)
        outs.append(out[:L])
    assert torch.equal(outs[0], outs[1])
    k, v = (p[tables[0].long()].transpose(1, 2).reshape(mb * 16, heads, hd)[:L].double().transpose(0, 1) for p in (kp, vp))
    s = torch.einsum("lhd,hkd->hlk", q[:L].double().reshape(L, heads, hd), k) * hd ** -0.5
    s.masked_fill_(torch.ones(L, L, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = torch.einsum("hlk,hkd->lhd", s.softmax(-1), v).reshape(L, -1)
    assert float((outs[0].double() - want).abs().max()) < 2e-5   # f32 sums of up to 465 terms


# The streaming RMSNorm reads everything behind its dependency wait: norm weights that the launch before it has just written (a GEMM whose
# dependents may start while it runs) are the new ones.
@pytest.mark.parametrize("size,hd", [(320, 0), (768, 64), (1024, 128)])
def test_rmsnorm_stream_weights_just_written(ak, torch_cuda, size, hd):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(size)
    x = torch.randn(3000, size, device="cuda", generator=g)
    a, wt = torch.randn(1, 8192, device="cuda", generator=g).bfloat16(), (0.01 * torch.randn(size, 8192, device="cuda", generator=g)).bfloat16()
    pos = torch.arange(3000, device="cuda", dtype=torch.int32) if hd else None
    y, want = (torch.empty(3000, size, device="cuda") for _ in range(2))
    w = torch.empty(size, device="cuda")
    ak.ops.gemm_bf16(a, wt, w, 1, size, 8192, ak.EPI_STORE_F32)
    torch.cuda.synchronize()
    ak.ops.rmsnorm_rope_residual(x, None, w, want, pos, 3000, size, 1e-5, hd, ak.AK_F32)
    for _ in range(10):
        w.fill_(float("nan"))
        torch.cuda.synchronize()
        ak.ops.gemm_bf16(a, wt, w, 1, size, 8192, ak.EPI_STORE_F32)
        ak.ops.rmsnorm_rope_residual(x, None, w, y, pos, 3000, size, 1e-5, hd, ak.AK_F32)
        assert torch.equal(y, want)


# SiLU in the GEMM's epilogue over its whole range of arguments, both kernels: to half an ulp of bf16 (at most 2^-8 of the value; the quotient
# itself is within 2^-16), and below 2e-36 where the denominator exp(-v) passes 2^126 (v < -87): there the result is 0.
@pytest.mark.parametrize("m", [64, 1100])
def test_gemm_silu_range(ak, torch_cuda, m):
    torch = torch_cuda
    n, k = 264, 8
    c = torch.linspace(-110.0, 110.0, m).bfloat16()
    d = torch.cat((torch.linspace(-1.0, 1.0, 200), torch.tensor([0.0, -0.0, 1e-30, -1e-30, 88.0, -88.0, 1000.0, -1000.0, 1e20, -1e20, 3e38, -3e38]),
                   torch.linspace(-0.01, 0.01, 52))).bfloat16()
    a, wt = torch.zeros(m, k, dtype=torch.bfloat16), torch.zeros(n, k, dtype=torch.bfloat16)
    a[:, 0], a[:, 1], wt[:, 0], wt[:, 1] = c, 1.0, 1.0, d
    out = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    ak.ops.gemm_bf16(a.cuda(), wt.cuda(), out, m, n, k, ak.EPI_SILU_BF16)
    v = (c.double()[:, None] + d.double()[None, :]).float().double()      # the sum in f32
    want = v / (1.0 + torch.exp(-v))
    err = (out.cpu().double() - want).abs()
    assert bool((err <= (2.0 ** -8 + 2.0 ** -16) * want.abs() + 2e-36).all())
    assert bool((out.cpu()[v < -90.0] == 0.0).all()) and not bool(out.isnan().any())
