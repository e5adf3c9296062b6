"""LSTM cells and attention steps at the sizes where the launch rule changes kernels or a kernel has a ragged edge: one column,
whole and broken groups of 8 and 128 columns, hidden sizes that fill no k-block, few and many row tiles, with and without the
feed-input operand; against a float64 cell / the CPU oracle's tolerances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# dtype id -> (relative, absolute) tolerance: 3xTF32, fp16 split, bf16, tf32
TOL = {4: (2e-5, 2e-5), 5: (2e-5, 2e-5), 1: (3e-2, 3e-2), 2: (1e-2, 1e-2)}


def sigmoid(x):
    return 1.0 / (1.0 + np.exp(-x))


@pytest.mark.parametrize("dtype", sorted(TOL))
@pytest.mark.parametrize("H,B", [(64, 1), (68, 3), (104, 9), (264, 16), (500, 17), (504, 33), (520, 64), (1000, 8), (1000, 24),
                                 (1000, 65), (1000, 127), (1000, 129), (2048, 40), (1024, 700)])
@pytest.mark.parametrize("feed", [0, 1])
def test_cell_edges(dtype, H, B, feed):
    import torch
    from zoph_rnn_b200 import api
    if dtype == 1 and H % 8:
        pytest.skip("bf16 needs a multiple of 8")
    rng = np.random.default_rng(H * 1000 + B)
    V = 50
    t = []
    for _ in range(4):
        t += [(rng.standard_normal(H * H) / np.sqrt(H)).astype(np.float32), (rng.standard_normal(H) * 0.1).astype(np.float32)]
    t.append(rng.uniform(-1, 1, H * V).astype(np.float32))
    t += [(rng.standard_normal(H * H) / np.sqrt(H)).astype(np.float32) for _ in range(8 if feed else 4)]
    layer = api.Input_To_Hidden_Layer(H, V, feed_input=bool(feed), dtype=dtype)
    layer.load_weights(t)
    ids = rng.integers(0, V, B).astype(np.int32)
    mask = (rng.random(B) > 0.2).astype(np.int32)
    h, c, q = (rng.uniform(-1, 1, (B, H)).astype(np.float32) for _ in range(3))

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a)).cuda()
    got_h, got_c = layer.forward_prop(dev(ids), dev(mask), dev(h.reshape(-1)), dev(c.reshape(-1)), dev(q.reshape(-1)) if feed else None)
    mat = [np.asarray(x, dtype=np.float64).reshape(-1, H).T for x in t]  # column-major H x H
    Wh, b, emb, M = [mat[2 * g] for g in range(4)], [t[2 * g + 1].astype(np.float64) for g in range(4)], mat[8], mat[9:13]
    x = emb[:, ids].T
    pre = []
    for g in range(4):  # i, f, g (c), o; the input matrices come as i, f, o, c
        k = (0, 1, 3, 2)[g]
        z = x @ M[k].T + h.astype(np.float64) @ Wh[g].T + b[g]
        if feed:
            z = z + q.astype(np.float64) @ mat[13 + k].T
        pre.append(z)
    cn = sigmoid(pre[1]) * c + sigmoid(pre[0]) * np.tanh(pre[2])
    hn = sigmoid(pre[3]) * np.tanh(cn)
    r, a = TOL[dtype]
    np.testing.assert_allclose(got_h.cpu().numpy().reshape(B, H), hn * mask[:, None], rtol=r, atol=a)
    np.testing.assert_allclose(got_c.cpu().numpy().reshape(B, H), cn * mask[:, None], rtol=r, atol=a)


@pytest.mark.parametrize("dtype,H,B,feed", [(5, 1000, 257, 1), (5, 1000, 456, 0), (5, 968, 700, 1), (5, 1024, 900, 0), (5, 1000, 1100, 1), (4, 1000, 300, 1),
                                            (4, 640, 1500, 0), (1, 1000, 700, 1), (1, 2048, 321, 0), (1, 1000, 900, 0), (2, 1000, 600, 0)])
def test_cells_on_pairs_of_ctas(dtype, H, B, feed):
    """Many columns: tiles of three, two and one accumulators, full and broken column tiles, an odd number of packed weight tiles."""
    test_cell_edges(dtype, H, B, feed)


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("n,m,k", [(2000, 700, 1000), (2100, 513, 1000), (4000, 300, 1500)])
def test_products_on_pairs_of_ctas(mode, n, m, k):
    import torch
    from zoph_rnn_b200 import api
    rng = np.random.default_rng(n + m + k)
    W, X = (rng.standard_normal((k, n)) * 0.1).astype(np.float32), rng.standard_normal((m, k)).astype(np.float32)
    C = api.gemm(torch.as_tensor(W).cuda().reshape(-1), torch.as_tensor(X).cuda().reshape(-1), n, m, k, mode).cpu().numpy().reshape(m, n)
    scale = np.linalg.norm(X.astype(np.float64), axis=1)[:, None] * np.linalg.norm(W.astype(np.float64), axis=0)[None, :]
    assert (np.abs(C - X.astype(np.float64) @ W.astype(np.float64)) / scale).max() < {1: 8e-3, 2: 1.5e-3, 3: 4e-6, 4: 4e-6}[mode]  # as the smaller products


@pytest.mark.parametrize("dtype", sorted(TOL))
@pytest.mark.parametrize("H,B", [(72, 1), (104, 9), (264, 16), (500, 17), (504, 33), (520, 64), (1000, 8), (1000, 65), (1000, 127), (1000, 129), (324, 200)])
def test_scoring_with_early_operands_edges(dtype, H, B):
    """A scoring pass with feed-input at the same edges: there every cell but the first, and the combiner, multiplies by operands that were
    complete earlier before it waits for its predecessor (the layer calls above have none).  Log-probabilities against the float64
    witness; three target steps, ragged sentences."""
    from oracle import ref_numpy
    from zoph_rnn_b200 import api, synth
    if dtype == 1 and H % 8:
        pytest.skip("bf16 needs a multiple of 8")
    cfg = synth.make_cfg(2, H, 60, 90, attention=2, feed_input=1)
    w = synth.make_weights(cfg, seed=H + B, dist="normal", scale=1 / np.sqrt(H))
    m = api.neuralMT_model(cfg, dtype=dtype)
    m.load_weights(w)
    src, tin, tout = synth.make_s2s_batch(60, 90, B, 1, 3, 2, 3, seed=B)
    got, _ = m.get_error(src, tin, tout)
    r, a = TOL[dtype]
    np.testing.assert_allclose(got, ref_numpy.score_batch(cfg, w, src, tin, tout), rtol=r, atol=a)


@pytest.mark.parametrize("dtype", [5, 1, 4])
@pytest.mark.parametrize("H,B", [(72, 1), (200, 12), (504, 40), (1000, 64), (1000, 130)])
@pytest.mark.parametrize("att", [1, 2])
def test_attention_step_edges(oracle, dtype, H, B, att):
    """The attention step in the tensor-core engines against the exact engine on the same inputs."""
    import torch
    from zoph_rnn_b200 import api
    rng = np.random.default_rng(H + B)
    S = 7
    w = [(rng.standard_normal(H * H) / np.sqrt(H)).astype(np.float32) for _ in range(2)]
    w += [(rng.standard_normal(H) * 0.05).astype(np.float32), (rng.standard_normal(H) * 0.1).astype(np.float32)]
    w += [(rng.standard_normal(H * H) / np.sqrt(H)).astype(np.float32) for _ in range(2)]
    lens = rng.integers(1, S + 1, B).astype(np.int32)
    hs, h = (torch.as_tensor(rng.uniform(-0.3, 0.3, n).astype(np.float32)).cuda() for n in (S * B * H, B * H))
    mask = torch.ones(B, dtype=torch.int32, device="cuda")
    out = {}
    for dt in (3, dtype):
        layer = api.attention_layer(H, 3, att_type=att, dtype=dt)
        layer.load_weights(w)
        layer.prep_minibatch_info(hs, S, B, torch.as_tensor(lens).cuda(), torch.as_tensor(S - lens).cuda())
        out[dt] = layer.forward_prop(h, mask).cpu().numpy()
    r, a = TOL[dtype]
    np.testing.assert_allclose(out[dtype], out[3], rtol=r, atol=a)


@pytest.mark.parametrize("beam", [1, 2, 15, 16, 32])
def test_ragged_batch_equals_single_sentences(beam):
    """A batch whose sentences stop at different steps, in any order: every sentence's hypotheses are those of decoding it alone."""
    from zoph_rnn_b200 import api, synth
    cfg = synth.make_cfg(2, 128, 300, 1100, attention=1, feed_input=1, D=3)
    m = api.neuralMT_model(cfg, dtype=api.F32_SIMT)
    m.load_weights(synth.make_weights(cfg, seed=11, scale=0.3))
    rng = np.random.default_rng(beam)
    srcs = [rng.integers(2, 300, n).astype(np.int32) for n in (3, 11, 1, 7, 11, 2, 5)]
    kw = dict(beam=beam, k_best=3, min_ratio=0.5, max_ratio=1.5, longest_sent=30, want_align=True)
    ids, ln, sc, al = m.decode(srcs, **kw)
    for i, s in enumerate(srcs):
        i1, l1, s1, a1 = m.decode([s], **kw)
        np.testing.assert_array_equal(ln[i], l1[0])
        np.testing.assert_array_equal(ids[i], i1[0])
        np.testing.assert_array_equal(al[i], a1[0])
        np.testing.assert_allclose(sc[i], s1[0], rtol=1e-5)


@pytest.mark.parametrize("dtype", [5, 1, 4, 2])
@pytest.mark.parametrize("H,V,N", [(64, 130, 1), (72, 257, 15), (200, 1000, 16), (504, 1281, 17), (1000, 40000, 12), (512, 20001, 63),
                                   (1000, 5000, 65), (264, 19001, 128), (264, 19001, 129), (504, 20000, 200), (800, 5003, 144), (800, 5003, 145), (800, 5003, 256), (800, 5003, 257)])
def test_vocabulary_projection_edges(dtype, H, V, N):
    """Best words, their log-probabilities and the target's, on both sides of the column count where the kernel changes."""
    import torch
    from zoph_rnn_b200 import api
    rng = np.random.default_rng(H + V + N)
    D = (rng.standard_normal((H, V)) * 2 / np.sqrt(H)).astype(np.float32)  # (column-major V x H)
    b = (rng.standard_normal(V) * 0.1).astype(np.float32)
    h = rng.uniform(-1, 1, (N, H)).astype(np.float32)
    layer = api.softmax_layer(V, H, dtype=dtype)
    layer.load_weights(D.reshape(-1), b)
    z = h.astype(np.float64) @ D.astype(np.float64) + b
    logp = z - (z.max(1, keepdims=True) + np.log(np.exp(z - z.max(1, keepdims=True)).sum(1, keepdims=True)))
    dh, k = torch.as_tensor(h.reshape(-1)).cuda(), 5
    r, a = {5: (1e-5, 2e-5), 4: (1e-5, 2e-5), 1: (2e-2, 4e-2), 2: (5e-3, 5e-3)}[dtype]
    val, idx = (t.cpu().numpy().reshape(N, k) for t in layer.topk(dh, k)[:2])
    np.testing.assert_allclose(val, np.take_along_axis(logp, idx.astype(np.int64), 1), rtol=r, atol=a)
    np.testing.assert_allclose(val, -np.sort(-logp, axis=1)[:, :k], rtol=r, atol=a)
    tgt = rng.integers(0, V, N).astype(np.int32)
    got = layer.compute_loss(dh, torch.as_tensor(tgt).cuda(), torch.ones(N, dtype=torch.int32, device="cuda"))
    np.testing.assert_allclose(got.cpu().numpy().reshape(-1), logp[np.arange(N), tgt], rtol=r, atol=a)


@pytest.mark.parametrize("H,n_sent,beam", [(504, 5, 9), (520, 9, 8), (1000, 2, 12)])
def test_ensemble_of_one_model_twice(H, n_sent, beam):
    """The models of an ensemble run side by side and their cells take half an SM, a lone model's take all of it: a model beside its copy finds
    the hypotheses that it finds alone (the mean of two equal distributions), scores within the rounding of log(mean(exp))."""
    from zoph_rnn_b200 import api, synth
    cfg = synth.make_cfg(2, H, 200, 1500, attention=2, feed_input=1)
    w = synth.make_weights(cfg, seed=H, dist="normal", scale=2 / np.sqrt(H))
    ms = []
    for _ in range(2):
        m = api.neuralMT_model(cfg, dtype=5)
        m.load_weights(w)
        ms.append(m)
    rng = np.random.default_rng(H + beam)
    srcs = [rng.integers(2, 200, n).astype(np.int32) for n in rng.integers(1, 9, n_sent)]
    kw = dict(beam=beam, k_best=1, min_ratio=0.5, max_ratio=1.5, longest_sent=30)
    one, two = ms[0].decode(srcs, **kw), api.decode_ensemble(ms, [srcs, srcs], **kw)
    np.testing.assert_array_equal(two[1], one[1])
    np.testing.assert_array_equal(two[0], one[0])
    np.testing.assert_allclose(two[2], one[2], rtol=1e-5)


def test_two_models_on_two_threads():
    """Models on streams of their own, worked on at the same time: small ones, whose cells' CTAs would fit an SM together, a large one, and
    a search whose cells and projection run on pairs.  Every result is the one of working alone."""
    import threading
    from zoph_rnn_b200 import api, synth
    jobs = []
    for k, (H, B, att) in enumerate([(128, 24, 2), (192, 40, 1), (1000, 100, 2)]):
        cfg = synth.make_cfg(2, H, 300, 900, attention=att, feed_input=1, D=3)
        m = api.neuralMT_model(cfg, dtype=5)
        m.load_weights(synth.make_weights(cfg, seed=H, dist="normal", scale=1 / np.sqrt(H)))
        batch = synth.make_s2s_batch(300, 900, B, 2, 6, 2, 6, seed=k)
        srcs = synth.make_decode_sources(300, 30, 2, 6, seed=k)
        jobs.append(lambda m=m, b=batch: m.get_error(*b)[0])
        if H == 1000:
            jobs.append(lambda m=m, s=srcs: m.decode(s, beam=12, k_best=1, min_ratio=0.5, max_ratio=1.5, longest_sent=20)[2])
    alone = [j() for j in jobs]
    got = [[] for _ in jobs]

    def work(i, members):
        for _ in range(10):
            for j in members:
                got[j].append(jobs[j]())
    threads = [threading.Thread(target=work, args=(i, mem)) for i, mem in enumerate([[0], [1], [2, 3]])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for j, a in enumerate(alone):
        assert len(got[j]) == 10
        for g in got[j]:
            np.testing.assert_array_equal(g, a)


@pytest.mark.parametrize("dtype,H,V,N", [(5, 336, 129, 65), (5, 336, 256, 96), (5, 324, 257, 97), (5, 320, 513, 513), (5, 1000, 3001, 700), (5, 600, 20000, 1025),
                                         (4, 104, 385, 160), (4, 324, 19001, 321), (1, 1024, 511, 160), (1, 1032, 2050, 289), (2, 544, 700, 255)])
def test_vocabulary_projection_pairs_of_ctas(dtype, H, V, N):
    """One and several column tiles, full and broken; a pair whose second CTA has no vocabulary row at all; both sides of the K where short
    log-sum-exp products leave the pairs; tiles of one and of two accumulator buffers."""
    test_vocabulary_projection_edges(dtype, H, V, N)


@pytest.mark.parametrize("mode,K,steps", [(4, 64, 4), (4, 320, 4), (4, 512, 4), (4, 1000, 8), (3, 64, 4), (3, 512, 4), (3, 1000, 8)])
@pytest.mark.parametrize("n,m", [(512, 100), (1000, 12), (320, 200)])
def test_products_of_one_sign_do_not_shrink(mode, K, steps, n, m):
    """The tensor core truncates: at each k-step the products, as they are aligned, and the new accumulator, which positive terms show as a
    shrinking sum.  Taken as one ulp per k-step (at most 2^-23 of a partial sum that grows linearly), an accumulator that absorbs `steps`
    of them loses (steps + 1) 2^-24 of its sum.  Adding the accumulators up in fp32, and storing, rounds: below 2^-24 on average."""
    import torch
    from zoph_rnn_b200 import api
    rng = np.random.default_rng(n + m + K)
    W, X = rng.uniform(0.05, 0.15, (K, n)).astype(np.float32), rng.uniform(0.5, 1.5, (m, K)).astype(np.float32)
    C = api.gemm(torch.as_tensor(W).cuda().reshape(-1), torch.as_tensor(X).cuda().reshape(-1), n, m, K, mode).cpu().numpy().reshape(m, n)
    want = X.astype(np.float64) @ W.astype(np.float64)
    assert np.abs(C / want - 1).mean() < (steps + 2) * 2.0 ** -24


@pytest.mark.parametrize("mode,K,steps", [(4, 320, 4), (4, 512, 4), (4, 1000, 8), (3, 320, 4), (3, 512, 4), (3, 1000, 8)])
@pytest.mark.parametrize("n,m", [(2000, 520), (3000, 400), (6000, 200)])
def test_products_of_one_sign_do_not_shrink_in_tiles_of_128_rows(mode, K, steps, n, m):
    """Which tile takes a product is a question of time: accumulators of the tiles of 128 x 128 absorb what those of the narrow ones do."""
    test_products_of_one_sign_do_not_shrink(mode, K, steps, n, m)


@pytest.mark.parametrize("mode,K", [(1, 1000), (1, 2000), (2, 500), (2, 1000), (2, 2000)])
@pytest.mark.parametrize("n,m", [(4000, 700), (4000, 1100)])
def test_single_pass_products_on_pairs_keep_two_accumulators(mode, K, n, m):
    """Operands that the mode holds exactly, all positive, of magnitudes that make no sum exact: what is missing from a result is what the tensor core has truncated, in proportion
    to the k-steps that an accumulator absorbs.  The first 200 columns alone take tiles of one CTA, whose two MMA warps have an
    accumulator each: a product of many columns, on pairs, loses no more (with one accumulator twice as much; 1.25 is for the other order of the k-steps)."""
    import torch
    from zoph_rnn_b200 import api
    rng = np.random.default_rng(n + m + K)
    W, X = [(np.exp2(rng.uniform(-6, 0, s)).astype(np.float32).view(np.uint32) & (0xffff0000 if mode == 1 else 0xffffe000)).astype(np.uint32).view(np.float32)
            for s in ((K, n), (m, K))]
    want = X.astype(np.float64) @ W.astype(np.float64)
    dW, dX = torch.as_tensor(W).cuda().reshape(-1), torch.as_tensor(X).cuda().reshape(-1)
    many, few = [1 - (api.gemm(dW, dX[:c * K], n, c, K, mode).cpu().numpy().reshape(c, n) / want[:c]).mean() for c in (m, 200)]
    assert few > 3 * 2.0 ** -24  # (it is seen at all)
    assert many < 1.25 * few


@pytest.mark.parametrize("K", [1000, 2000])
@pytest.mark.parametrize("m", [250, 400, 700, 900])
def test_tf32_products_absorb_a_quarter_of_the_k_axis_in_every_tile(K, m):
    """As above: 128 columns take tiles split over two CTAs with two accumulators each.  Tiles of 64 and of 128 rows on one CTA and pairs of CTAs
    (250, 400, 700 and 900 columns) lose no more."""
    import torch
    from zoph_rnn_b200 import api
    rng = np.random.default_rng(m + K)
    n = 4000
    W, X = [(np.exp2(rng.uniform(-6, 0, s)).astype(np.float32).view(np.uint32) & 0xffffe000).astype(np.uint32).view(np.float32) for s in ((K, n), (m, K))]
    want = X.astype(np.float64) @ W.astype(np.float64)
    dW, dX = torch.as_tensor(W).cuda().reshape(-1), torch.as_tensor(X).cuda().reshape(-1)
    many, few = [1 - (api.gemm(dW, dX[:c * K], n, c, K, 2).cpu().numpy().reshape(c, n) / want[:c]).mean() for c in (m, 128)]
    assert few > 3 * 2.0 ** -24  # (it is seen at all)
    assert many < 1.25 * few


@pytest.mark.parametrize("dtype", [5, 4, 1])
@pytest.mark.parametrize("H,V", [(504, 3000), (1000, 700), (104, 9000)])
def test_vocabulary_projection_with_values_that_are_not_finite(dtype, H, V):
    """Logits of -inf (words that are masked out by their bias), NaN and infinite hidden states, in launches of many columns on pairs of CTAs
    and on single ones: a column shows what its own states and the biases make of it, as in a launch of few columns, whatever the others hold."""
    import torch
    from zoph_rnn_b200 import api
    g = torch.Generator(device="cuda").manual_seed(H + V)
    D = ((torch.rand(V * H, generator=g, device="cuda") - .5) * .4).cpu().numpy()
    bias = ((torch.rand(V, generator=g, device="cuda") - .5) * .4).cpu().numpy()
    bias[[0, 5, 64, V - 1]] = -np.inf
    bias[128:192] = -np.inf  # (whole parts)
    h = torch.tanh(torch.randn(1200 * H, generator=g, device="cuda")).view(1200, H)
    targets = torch.randint(200, V - 1, (1200,), generator=g, device="cuda", dtype=torch.int32)
    targets[3] = 5
    for nan_word in (None, 300):
        b = bias.copy()
        if nan_word is not None:
            b[nan_word] = np.nan
        s = api.softmax_layer(V, H, dtype=dtype)
        s.load_weights(D, b)
        for N in (100, 300, 1200):
            x, t = h[:N].clone(), targets[:N].contiguous()
            mask = torch.ones(N, dtype=torch.int32, device="cuda")
            clean = [s.compute_loss(x.reshape(-1), t, mask).cpu().numpy().reshape(-1)] + [a.cpu().numpy().reshape(N, -1) for a in s.topk(x.reshape(-1), 13)[:2]]
            few = [s.compute_loss(x[:40].reshape(-1), t[:40], mask[:40]).cpu().numpy().reshape(-1)] + [a.cpu().numpy().reshape(40, -1) for a in s.topk(x[:40].reshape(-1), 13)[:2]]
            # the kernels add in another order
            np.testing.assert_allclose(clean[0][:40], few[0], rtol=2e-6, atol=2e-6)
            np.testing.assert_allclose(clean[1][:40], few[1], rtol=2e-6, atol=2e-6)
            if nan_word is None:
                assert clean[0][3] == -np.inf and np.isfinite(clean[0][np.arange(N) != 3]).all() and np.isfinite(clean[1]).all()
                assert not np.isin(clean[2], np.r_[[0, 5, 64, V - 1], 128:192]).any()
            else:
                assert np.isnan(clean[0][np.arange(N) != 3]).all()
            x[7, 1], x[33, 2], x[N - 1, :] = float("nan"), float("inf"), float("nan")
            bad, rest = [7, 33, N - 1], np.setdiff1d(np.arange(N), [7, 33, N - 1])
            got = [s.compute_loss(x.reshape(-1), t, mask).cpu().numpy().reshape(-1)] + [a.cpu().numpy().reshape(N, -1) for a in s.topk(x.reshape(-1), 13)[:2]]
            for a, c in zip(got, clean):
                np.testing.assert_array_equal(a[rest], c[rest])
            assert not np.isfinite(got[0][bad]).any()


@pytest.mark.parametrize("H,B", [(600, 44), (640, 36), (1200, 28)])
def test_cells_of_a_few_more_columns_are_as_close_to_float64(H, B):
    """Where the launch rule leaves the warp-level kernel for links is a question of precision, too: at these sizes links, whose accumulators absorb
    four times as many products, are 27 % farther from float64 than a launch of 16 columns, which the warp-level kernel takes."""
    import torch
    from zoph_rnn_b200 import api
    g = torch.Generator(device="cuda").manual_seed(H)
    w = []
    for _ in range(4):
        w += [(torch.rand(H * H, generator=g, device="cuda") - .5) * .16, torch.zeros(H, device="cuda")]
    w += [(torch.rand(H * H, generator=g, device="cuda") - .5) * .16 for _ in range(4)]
    layer = api.Hidden_To_Hidden_Layer(H, dtype=5)
    layer.load_weights([t.cpu().numpy() for t in w])
    mat = [t.double().view(-1, H).t() for t in w]  # W_hi b_i W_hf b_f W_hc b_c W_ho b_o M_i M_f M_o M_c

    def distance(cols):
        err = ref = 0.0
        for _ in range(8):
            x, h, c = [torch.tanh(torch.randn(H * cols, generator=g, device="cuda")) for _ in range(3)]
            got, _ = layer.forward_prop(x, torch.ones(cols, dtype=torch.int32, device="cuda"), h, c)
            X, Hh, C = [t.double().view(cols, H) for t in (x, h, c)]
            i, f, gg, o = [X @ mat[8 + (0, 1, 3, 2)[k]].t() + Hh @ mat[2 * k].t() for k in range(4)]
            want = torch.sigmoid(o) * torch.tanh(torch.sigmoid(f) * C + torch.sigmoid(i) * torch.tanh(gg))
            err += ((got.double().view(cols, H) - want) ** 2).sum().item()
            ref += (want ** 2).sum().item()
        return (err / ref) ** 0.5
    assert distance(B) < 1.1 * distance(16)
