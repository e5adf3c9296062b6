"""The work that users of this library have it do, as cases that can be timed: teacher-forced scoring (`get_error`), beam
decoding (`decode`, `decode_ensemble`) and one target step through the layer objects, each through its public entry point.
Sizes are the benchmark configurations' and the tests', and generic ones between them.  Scoring and decoding take host
arrays and give host arrays, as the front end calls them; the layer step works on device tensors.

A case's model keeps its weights for as long as the case is worked on, as a program that scores or decodes a stream of
minibatches does; the minibatches (ids, lengths, states) come from the seed.
"""
import numpy as np
import torch

from zoph_rnn_b200 import api, synth

_BYTES = {"f32": 4, "bf16": 2}
_DTYPE = {"f32": api.F32, "bf16": api.BF16}


# ------------------------------------------------------------------------------------------------ the cases
def _score(name, layers, H, Vs, Vt, B, S, T, att=0, feed=0, dtype="f32", scale=0.1, zipf=1.1):
    """S, T: shortest and longest source / target sentence of the minibatch ((0, 0) source: a language model)."""
    return dict(name=name, kind="score", layers=layers, H=H, Vs=Vs, Vt=Vt, B=B, s_min=S[0], s_max=S[1], t_min=T[0], t_max=T[1],
                att=att, feed=feed, dtype=dtype, scale=scale, zipf=zipf)


def _decode(name, layers, H, Vs, Vt, B, S, beam, att, feed, k_best=1, align=False, models=1, ratio=2.0):
    return dict(name=name, kind="decode", layers=layers, H=H, Vs=Vs, Vt=Vt, B=B, s_min=S[0], s_max=S[1], beam=beam, att=att,
                feed=feed, k_best=k_best, align=align, models=models, ratio=ratio, dtype="f32", scale=0.06, zipf=1.1)


def _layers(name, layers, H, V, B, S, k, att, feed, dtype="f32"):
    return dict(name=name, kind="layers", layers=layers, H=H, Vs=V, Vt=V, B=B, s_min=max(1, S // 3), s_max=S, k=k, att=att,
                feed=feed, dtype=dtype, scale=0.1, zipf=1.1)


def listed():
    return [
        # a small language model on short minibatches: the shortest call there is, bound by latency
        _score("lm_small", 1, 100, 0, 10000, 8, (0, 0), (35, 35), scale=0.08, zipf=0.0),
        # a large-vocabulary language model with bf16 weights: the largest matrix products
        _score("lm_large_bf16", 2, 2048, 0, 200000, 256, (0, 0), (64, 64), dtype="bf16", scale=0.035, zipf=1.05),
        # scoring of a test set in full minibatches with the deep attention model, in both arithmetics
        _score("score_global", 4, 1000, 50000, 50000, 128, (50, 50), (50, 50), att=2, feed=1),
        _score("score_global_bf16", 4, 1000, 50000, 50000, 128, (50, 50), (50, 50), att=2, feed=1, dtype="bf16"),
        # the local-p model of the original program on ragged sources
        _score("score_localp", 2, 1000, 40000, 40000, 64, (10, 80), (60, 60), att=1, feed=1),
        # force-decoding sentence by sentence (minibatch 1), as n-best rescoring of one sentence does
        _score("score_single", 2, 1000, 40000, 40000, 1, (27, 27), (25, 25), att=1, feed=1),
        # a plain encoder-decoder without attention, sizes that fill no tile, ragged on both sides
        _score("score_plain", 3, 500, 20000, 20000, 50, (3, 47), (4, 45)),
        # beam decoding of a file in batches of sentences of all lengths
        _decode("decode_batch", 2, 1000, 50000, 50000, 64, (10, 50), 12, att=2, feed=1),
        # interactive translation: one sentence, the default beam
        _decode("decode_single", 2, 1000, 40000, 40000, 1, (23, 23), 12, att=1, feed=1, ratio=1.5),
        # n-best lists with alignments for <UNK> replacement
        _decode("decode_nbest", 2, 500, 20000, 20000, 20, (4, 40), 10, att=1, feed=1, k_best=4, align=True, ratio=1.5),
        # an ensemble of two models
        _decode("decode_ensemble", 2, 500, 20000, 20000, 9, (8, 30), 8, att=2, feed=1, models=2, ratio=1.5),
        # a host program that drives the layer objects itself: one target step of a beam
        _layers("layer_step", 2, 1000, 50000, 12, 30, 13, att=2, feed=1),
    ]


_LARGEST = {"score": 16e12, "decode": 6.8e12, "layers": 1e12}  # operations of the largest listed cases, about


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))))


def _hidden(rng, lo, hi, dtype):
    step = 8 if dtype == "bf16" else 4  # what the tensor-core engines take
    return max(step, _log_int(rng, lo, hi) // step * step)


def draw(rng):
    while True:
        c = _draw(rng)
        if _cost(c) <= _LARGEST[c["kind"]]:
            c.pop("name")
            return c


def _draw(rng):
    what = rng.choice(["lm_small", "lm", "s2s", "s2s", "plain", "single", "decode", "decode", "decode_single", "ensemble", "layers", "layers"])
    dtype = rng.choice(["f32", "f32", "bf16"])
    if what == "lm_small":  # any hidden size: the small layers have kernels of their own
        return _score("", rng.choice([1, 2]), _log_int(rng, 40, 300), 0, _log_int(rng, 1000, 30000), _log_int(rng, 1, 32), (0, 0),
                      (1, _log_int(rng, 8, 60)), scale=0.08)
    if what == "lm":
        V = _log_int(rng, 5000, 200000)
        return _score("", rng.choice([1, 2, 3]), _hidden(rng, 320, 2048, dtype), 0, V, _log_int(rng, 8, 256), (0, 0),
                      (rng.choice([3, 20]), _log_int(rng, 20, 64)), dtype=dtype, scale=0.05, zipf=1.05)
    H, V = _hidden(rng, 256, 1024, dtype), _log_int(rng, 5000, 50000)
    L = rng.choice([1, 2, 3, 4])
    att = rng.choice([1, 2])
    if what == "s2s":
        return _score("", L, H, V, _log_int(rng, 5000, 50000), _log_int(rng, 8, 200), (rng.choice([2, 10]), _log_int(rng, 16, 80)),
                      (rng.choice([3, 12]), _log_int(rng, 16, 80)), att=att, feed=rng.choice([1, 1, 0]), dtype=dtype)
    if what == "plain":
        return _score("", L, H, V, _log_int(rng, 5000, 50000), _log_int(rng, 8, 200), (2, _log_int(rng, 16, 80)),
                      (3, _log_int(rng, 16, 80)), dtype=dtype)
    if what == "single":
        S, T = _log_int(rng, 5, 80), _log_int(rng, 5, 80)
        return _score("", L, H, V, V, rng.choice([1, 1, 2, 5]), (S, S), (T, T), att=rng.choice([0, 1, 2]), feed=1, dtype=dtype)
    H = _hidden(rng, 256, 1024, "f32")
    L = min(L, 3)
    if what == "decode":
        return _decode("", L, H, V, V, _log_int(rng, 4, 64), (rng.choice([3, 8]), _log_int(rng, 12, 50)), rng.randint(2, 16),
                       att=rng.choice([0, 1, 2]), feed=1, k_best=rng.choice([1, 1, 3]), ratio=rng.choice([1.5, 2.0]))
    if what == "decode_single":
        S = _log_int(rng, 5, 60)
        return _decode("", L, H, V, V, 1, (S, S), rng.choice([1, 5, 8, 12, 15]), att=att, feed=1, align=rng.choice([False, True]), ratio=1.5)
    if what == "ensemble":
        return _decode("", min(L, 2), H, V, V, _log_int(rng, 1, 16), (4, _log_int(rng, 8, 30)), rng.randint(3, 12), att=att, feed=1,
                       align=rng.choice([False, True]), models=rng.choice([2, 3]), ratio=1.5)
    if dtype == "bf16":
        H = H // 8 * 8
    return _layers("", L, H, V, _log_int(rng, 1, 256), _log_int(rng, 8, 60), 13, att=att, feed=rng.choice([0, 1]), dtype=dtype)


# ------------------------------------------------------------------------------------------------ weights and inputs
_kept = {}  # the model (or layers) of the case being worked on


def _config(case):
    lm = int(case["s_max"] == 0)
    return synth.make_cfg(case["layers"], case["H"], case["Vs"], case["Vt"], lm=lm, attention=case["att"],
                          feed_input=case["feed"] if case["att"] else 0, D=10)


def _tensor(gen, n, scale):
    return (torch.rand(n, generator=gen, device="cuda") * (2 * scale) - scale).cpu().numpy()


def _weights(cfg, case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for name, r, c in synth.tensor_spec(cfg):
        scale = case["scale"]
        if case["kind"] != "score" and name == "softmax.D":
            scale = 2.0  # a decoder's model has been trained: it is fairly sure of its next word
        out.append(_tensor(gen, r * c, scale))
    return out


def _model(case):
    """The case's models or layer objects; those of the case before are let go."""
    key = tuple(sorted((k, v) for k, v in case.items() if k in ("kind", "layers", "H", "Vs", "Vt", "att", "feed", "dtype", "scale", "models", "s_max")))
    if key not in _kept:
        _kept.clear()
        cfg = _config(case)
        dtype = _DTYPE[case["dtype"]]
        if case["kind"] == "layers":
            _kept[key] = _layer_objects(case, cfg, dtype)
        else:
            got = []
            for k in range(case.get("models", 1)):
                m = api.neuralMT_model(cfg, dtype=dtype)
                m.load_weights(_weights(cfg, case, 1234 + k))
                got.append(m)
            _kept[key] = got
    return _kept[key]


def _layer_objects(case, cfg, dtype):
    w = dict(zip([n for n, _, _ in synth.tensor_spec(cfg)], _weights(cfg, case, 1234)))
    stack = []
    for l in range(case["layers"]):
        if l == 0:
            layer = api.Input_To_Hidden_Layer(case["H"], case["Vt"], feed_input=bool(cfg["feed_input"]), dtype=dtype)
        else:
            layer = api.Hidden_To_Hidden_Layer(case["H"], dtype=dtype)
        layer.load_weights([t for n, t in w.items() if n.startswith("tgt%d." % l)])
        stack.append(layer)
    att = api.attention_layer(case["H"], 10, att_type=case["att"], dtype=dtype)
    att.load_weights([t for n, t in w.items() if n.startswith("att.")])
    soft = api.softmax_layer(case["Vt"], case["H"], dtype=dtype)
    soft.load_weights(w["softmax.D"], w["softmax.b_d"])
    return dict(stack=stack, att=att, soft=soft)


def _lengths(lo, hi, n):
    """n sentence lengths spread evenly over lo .. hi, the longest among them."""
    if n == 1:
        return np.array([hi])
    return np.round(np.linspace(lo, hi, n)).astype(np.int64)


def _sampler(V, zipf, seed):
    if zipf:
        return synth.zipf_sampler(V, zipf, seed)
    return lambda gen, n: gen.integers(0, V, size=n, dtype=np.int32)


def prepare(case, seed):
    state = dict(case=case, model=_model(case))
    gen = np.random.default_rng(seed)
    B = case["B"]
    if case["kind"] == "layers":
        return _prepare_layers(state, case, gen, seed)
    if case["s_max"]:
        s_len = gen.permutation(_lengths(case["s_min"], case["s_max"], B))
        words = _sampler(case["Vs"], case["zipf"], seed + 1)
        sources = [words(gen, n).astype(np.int32) for n in s_len]
    if case["kind"] == "decode":
        state["sources"] = sources
        return state
    # a minibatch in the original program's layout: time-major, sources reversed and padded on the left with -1, targets
    # <START> y1 .. yn and y1 .. yn <EOF> padded on the right
    t_len = gen.permutation(_lengths(case["t_min"], case["t_max"], B))
    words = _sampler(case["Vt"] - 2, case["zipf"], seed + 2)
    tin = np.full((case["t_max"], B), -1, dtype=np.int32)
    tout = tin.copy()
    for b, n in enumerate(t_len):
        y = words(gen, n - 1) + 2
        tin[0, b] = 0
        tin[1:n, b] = y
        tout[: n - 1, b] = y
        tout[n - 1, b] = 1
    src = None
    if case["s_max"]:
        src = np.full((case["s_max"], B), -1, dtype=np.int32)
        for b, s in enumerate(sources):
            src[case["s_max"] - len(s):, b] = s
    state.update(src=src, tin=tin, tout=tout)
    return state


def _prepare_layers(state, case, gen, seed):
    H, B, S = case["H"], case["B"], case["s_max"]
    tgen = torch.Generator(device="cuda").manual_seed(seed)

    def hidden(n):  # states of an LSTM: within -1 .. 1, most of them small
        return torch.tanh(0.5 * torch.randn(n, generator=tgen, device="cuda"))

    lens = gen.permutation(_lengths(case["s_min"], S, B)).astype(np.int32)
    words = _sampler(case["Vt"], case["zipf"], seed + 1)
    state.update(
        ids=torch.as_tensor(words(gen, B).astype(np.int32)).cuda(), mask=torch.ones(B, dtype=torch.int32, device="cuda"),
        h=[hidden(H * B) for _ in range(case["layers"])], c=[2 * hidden(H * B) for _ in range(case["layers"])],
        htild=hidden(H * B) if case["feed"] else None, hs=hidden(S * B * H), lens=torch.as_tensor(lens).cuda(),
        offsets=torch.as_tensor(S - lens).cuda())
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    case, model = state["case"], state["model"]
    if case["kind"] == "score":
        return model[0].get_error(state["src"], state["tin"], state["tout"])
    if case["kind"] == "decode":
        kw = dict(beam=case["beam"], k_best=case["k_best"], min_ratio=0.5, max_ratio=case["ratio"], longest_sent=100,
                  want_align=bool(case["align"]))
        if case["models"] > 1:
            return api.decode_ensemble(model, [state["sources"]] * case["models"], **kw)
        return model[0].decode(state["sources"], **kw)
    hs, cs = [], []
    for l, layer in enumerate(model["stack"]):
        if l == 0:
            h, c = layer.forward_prop(state["ids"], state["mask"], state["h"][0], state["c"][0], state["htild"])
        else:
            h, c = layer.forward_prop(hs[-1], state["mask"], state["h"][l], state["c"][l])
        hs.append(h)
        cs.append(c)
    att = model["att"]
    att.prep_minibatch_info(state["hs"], case["s_max"], case["B"], state["lens"], state["offsets"])
    htild = att.forward_prop(hs[-1], state["mask"])
    return hs, cs, htild, model["soft"].topk(htild, case["k"])


# ------------------------------------------------------------------------------------------------ what a pass needs
def _totals(case):
    """(source words, target columns computed, weight values read, embedding rows read) of one pass, padding left out."""
    H, L, B = case["H"], case["layers"], case["B"]
    HH = H * H
    feed = case["feed"] and case["att"]
    cell_w = 8 * HH * L + (4 * HH if feed else 0)
    att_w = {0: 0, 1: 4 * HH, 2: 2 * HH}[case["att"]]
    src = int(_lengths(case["s_min"], case["s_max"], B).sum()) if case["s_max"] else 0
    if case["kind"] == "score":
        tgt = int(_lengths(case["t_min"], case["t_max"], B).sum())
    elif case["kind"] == "decode":
        beam = min(case["beam"], int(case["Vt"] ** 0.5))
        tgt = sum(1 + beam * min(int(case["ratio"] * n), 102) for n in _lengths(case["s_min"], case["s_max"], B))
    else:
        src, tgt = 0, B
    weights = cell_w + att_w + case["Vt"] * H + (8 * HH * L if src else 0)
    macs = src * 8 * HH * L + tgt * (cell_w + att_w + case["Vt"] * H)
    if case["att"]:  # scores and context over the sentence or over the window
        mean_s = float(_lengths(case["s_min"], case["s_max"], B).mean())
        macs += tgt * 2 * H * min(mean_s, 21 if case["att"] == 1 else mean_s)
    return src, tgt, weights, macs


def _cost(case):
    return 2.0 * _totals(case)[3] * case.get("models", 1)


def work(case):
    eb, K, H, B = _BYTES[case["dtype"]], case.get("models", 1), case["H"], case["B"]
    src, tgt, weights, macs = _totals(case)
    if case["kind"] == "decode":
        rows = src + min(tgt, case["Vt"])
        io = 4 * src + B * case["k_best"] * (104 * (2 if case["align"] else 1) + 2) * 4
    elif case["kind"] == "score":
        rows = min(src, case["Vs"]) + min(tgt, case["Vt"])
        io = 4 * (src + 3 * tgt)
    else:
        L = case["layers"]
        rows = B
        io = 4 * (H * B * (4 * L + 1 + (1 if case["feed"] else 0)) + 2 * B * case["k"] + 5 * B)
        io += 4 * H * int(np.minimum(_lengths(case["s_min"], case["s_max"], B), 21 if case["att"] == 1 else 10**9).sum())
    return {"bytes": float(K * eb * (weights + H * rows) + io), "flops": 2.0 * K * macs}


def tolerance(case):
    if case["kind"] == "decode":
        # words, lengths, alignments and scores of the best hypotheses: scores as 32-bit sums over the steps; a word differs
        # where two hypotheses tie within rounding, which takes the rest of its row along
        return {"rel": 3e-4, "max": 2e-2, "differ": 0.01}
    if case["dtype"] == "bf16":  # operands rounded to bf16 at every step
        return {"rel": 1e-2, "max": 0.2, "differ": 0.01}
    if case["att"] == 1:
        # local-p attention cuts its window at int(p_t): where p_t lies within rounding of a whole number, a window moves by
        # one position and the rest of that sentence with it
        return {"rel": 5e-4, "max": 5e-2, "differ": 0.01}
    return {"rel": 1e-5, "max": 4e-4, "differ": 0.01}  # whole values: two words of a candidate list may swap places
