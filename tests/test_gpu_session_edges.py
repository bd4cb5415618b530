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


# Generation that ends at an end-of-sequence token: decode steps (and samplers) were launched past it and have written cache rows beyond
# cur_len. The same session then goes on as if they had never run: a decode step, a second generate, a generate on a new cache.
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("sampler", [{}, dict(temperature=0.9, top_k=12, top_p=0.95, repetition_penalty=1.1, seed=5)])
@pytest.mark.parametrize("cfg_args", [(40, 64, 1, 1, 64), (40, 60, 1, 1, 64)])   # the persistent step; the launch chain (head_dim 60)
def test_session_goes_on_after_an_early_stop(ak, ctx, cfg_args, sampler, dtype):
    if dtype == 1 and cfg_args[1] == 60:
        cfg_args = (40, 32, 1, 1, 64)   # (bf16 wants a width of whole 16-byte vectors)
    params = ak.synthetic_weights(ak.ModelConfig(*cfg_args), seed=3, std=0.3)
    prompt, more = ak.uniform_tokens(5, 40, seed=1), ak.uniform_tokens(3, 40, seed=2)
    N = 40
    free = ak.ModelConfig(*cfg_args)
    w = ak.ModelWeights.from_params(ctx, free, params, dtype)
    s = ak.InferenceSession(ctx, w, 64)
    full = s.generate(prompt, N, stop_on_eos=False, **sampler).tolist()
    s.close(); w.close()
    # the tokens whose first appearance is at the start, a little later, and in the middle
    stops = [full[0]] + [t for i, t in enumerate(full) if t not in full[:i] and 0 < i < N - 1][:3]
    assert len(stops) >= 2
    for eos in stops:
        cfg = ak.ModelConfig(*cfg_args, eos_token=int(eos))
        w = ak.ModelWeights.from_params(ctx, cfg, params, dtype)
        s, ref = ak.InferenceSession(ctx, w, 64), ak.InferenceSession(ctx, w, 64)
        first = full.index(eos)
        out = s.generate(prompt, N, stop_on_eos=True, **sampler)
        assert out.tolist() == full[:first + 1]
        assert s.cur_len == prompt.size + first          # the last token is not in the cache
        # a session that was only given the tokens
        ref.replace_cache()
        ref.prefill(prompt)
        for t in out[:-1]:
            ref.decode_step(int(t))
        for layer in range(cfg.num_layers):
            for a, b in zip(s.read_cache(layer), ref.read_cache(layer)):
                assert np.array_equal(a, b)
        for t in more:
            (ga, ta), (gb, tb) = s.decode_step(int(t)), ref.decode_step(int(t))
            assert np.array_equal(ga, gb) and ta == tb
        assert np.array_equal(s.generate(more, 9, stop_on_eos=True, **sampler), ref.generate(more, 9, stop_on_eos=True, **sampler))
        assert s.cur_len == ref.cur_len
        s.replace_cache()
        assert s.generate(prompt, N, stop_on_eos=False, **sampler).tolist() == full
        s.close(); ref.close(); w.close()
    ctx.check_device_status()


# The context fills before max_new: one token more than there are steps, whether the steps run ahead or not.
@pytest.mark.parametrize("sampler", [{}, dict(temperature=0.9, top_k=12, top_p=0.95, repetition_penalty=1.1, seed=5)])
@pytest.mark.parametrize("max_ctx,max_new,tokens,cur", [(20, 100, 16, 20), (20, 16, 16, 20), (20, 15, 15, 20), (20, 14, 14, 19), (5, 3, 1, 5), (20, 0, 0, 5)])
def test_generate_fills_the_context(ak, ctx, sampler, max_ctx, max_new, tokens, cur):
    cfg = ak.ModelConfig(40, 64, 1, 1, 64)
    w = ak.ModelWeights.from_params(ctx, cfg, ak.synthetic_weights(cfg, seed=3, std=0.3), 0)
    s = ak.InferenceSession(ctx, w, max_ctx)
    out = s.generate(ak.uniform_tokens(5, 40, seed=1), max_new, stop_on_eos=False, **sampler)
    assert len(out) == tokens and s.cur_len == cur
    s.close(); w.close()


# f32: a prompt's row has the same bits whether it is prefilled alone or with others (one token: one row in the launch), in a session and
# in an engine with and without the padding of captured steps.
@pytest.mark.parametrize("dim,heads,ffn", [(320, 5, 1280), (768, 12, 3072)])
def test_one_token_prompt_f32(ak, ctx, dim, heads, ffn):
    cfg = ak.ModelConfig(500, dim, heads, 3, 64, ffn)
    w = ak.ModelWeights(ctx, cfg, ak.AK_F32)
    w.init_synthetic(3, 0.05)
    rows = []
    for n in (1, 2, 40):
        s = ak.InferenceSession(ctx, w, 64)
        s.replace_cache()
        s.prefill(np.arange(7, 7 + n, dtype=np.uint32))
        rows.append([a[0].copy() for layer in range(3) for a in s.read_cache(layer)])
        s.close()
    for other in rows[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(rows[0], other))
    outs = []
    for prompts, graph in (([[7]], False), ([[7]], True), ([[7], [9, 11, 13]], False)):
        e = ak.Engine(ctx, w, max_seqs=3, max_seq_len=48, use_cuda_graph=graph)
        ids = [e.submit(p, 48) for p in prompts]
        e.run_to_completion()
        outs.append(e.poll(ids[0])[0].tolist())
        e.close()
    assert outs[0] == outs[1] == outs[2]
    w.close()


# A residual stream whose squares overflow f32: the norm's factor is 0 (1 / sqrt(inf)), so every logit is 0, in the step as in a prefill.
@pytest.mark.parametrize("dtype", [0, 1])
def test_step_with_an_overflowing_norm(ak, ctx, dtype):
    cfg = ak.ModelConfig(200, 128, 2, 2, 64)
    params = ak.synthetic_weights(cfg, seed=1, std=0.05)
    params[0] = params[0] * np.float32(1e22)
    w = ak.ModelWeights.from_params(ctx, cfg, params, dtype)
    s = ak.InferenceSession(ctx, w, 64)
    s.replace_cache()
    want, tok = s.prefill([3, 4, 5])
    assert tok == 0 and np.array_equal(want, np.zeros(200, np.float32))
    got, tok = s.decode_step(6)
    assert tok == 0 and np.array_equal(got, want)
    s.close(); w.close()


# Two sessions on two contexts (streams) and an engine on a third, each in a thread of its own: a decode step needs every SM at once, the
# others' kernels take them meanwhile. Every thread gets the tokens that it gets alone.
def test_sessions_and_engine_in_threads(ak, ctx):
    import threading
    cfg = ak.ModelConfig(1000, 320, 5, 3, 256, 1280)
    ctxs = [ak.Context(0) for _ in range(3)]
    ws = [ak.ModelWeights(c, cfg, dt) for c, dt in zip(ctxs, (0, 1, 1))]
    for w in ws:
        w.init_synthetic(4, 0.05)
    prompts = [ak.uniform_tokens(9 + 5 * i, 1000, seed=i) for i in range(6)]

    def session(i):
        s = ak.InferenceSession(ctxs[i], ws[i], 256)
        out = []
        for p in prompts[:4]:
            s.replace_cache()
            out.append(s.generate(p, 60, stop_on_eos=False).tolist())
            s.replace_cache()
            out.append(s.generate(p, 40, stop_on_eos=False, temperature=0.8, top_k=20, top_p=0.9, repetition_penalty=1.1, seed=i).tolist())
        s.close()
        return out

    def engine(i):
        e = ak.Engine(ctxs[i], ws[i], max_seqs=4, max_seq_len=128, use_cuda_graph=True)
        out = []
        for _ in range(3):
            ids = [e.submit(p, 120) for p in prompts]
            e.run_to_completion()
            out += [e.poll(k)[0].tolist() for k in ids]
            e.clear_finished()
        e.close()
        return out

    jobs = [lambda: session(0), lambda: session(1), lambda: engine(2)]
    alone = [j() for j in jobs]
    for _ in range(2):
        got, errors = [None] * 3, []

        def work(k):
            try:
                got[k] = jobs[k]()
            except Exception as e:   # noqa: BLE001
                errors.append(e)
        threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        assert got == alone
    for c in ctxs:
        c.check_device_status()
    for w in ws:
        w.close()
    for c in ctxs:
        c.close()
