"""Layered decoders on the GPU against the plain restatement in layered_oracle.py: every mechanism alone, prompts, portions,
decoding, window and chunk edges, far keys, odd sizes, re-used sequences, and generation through the session layer."""
import copy
import json

import numpy as np
import pytest

import layered_oracle as lo
from kmll_b200 import pefisun, registry
from kmll_b200 import runtime as rt
from kmll_b200.checkpoint import write_safetensors
from kmll_b200.lib import KmllError, load
from kmll_b200.session import GenerationOptions, SamplingOptions, Session

pytestmark = pytest.mark.gpu

# relative to the root mean square of the logits (or of the residual stream), per position; bf16: activations of the projections
TOL = {"float32": 3e-5, "bfloat16": 4e-2}
DTYPES = ["float32", "bfloat16"]


def retention(heads=2, dim=16, vdim=24, decay=None, rot=None, base=400.0):
    return {"type": "retention", "mixer": {"heads": heads, "dim": dim, "vdim": vdim, "decay": decay or [0.93 + 0.06 * i / heads for i in range(heads)],
                                           "rot": {"base": base, "dims": dim if rot is None else rot}}, "mlp": None}


def lightning(heads=2, dim=24, vdim=16, decay=None):
    return {"type": "lightning", "mixer": {"heads": heads, "dim": dim, "vdim": vdim, "decay": decay or [0.8 + 0.19 * i / heads for i in range(heads)]},
            "mlp": None}


def latent(heads=3, dim=16, rot_dim=8, vdim=24, kv_rank=40, window=11, scale=0.2, scaling=None, base=3000.0):
    rot = {"base": base, "dims": rot_dim}
    if scaling:
        rot["scaling"] = scaling
    return {"type": "latent_attention", "mixer": {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": vdim, "kv_rank": kv_rank, "scale": scale,
                                                  "mask": {"size": window}, "rot": rot}, "mlp": None}


def with_mlp(layer, ff):
    return {**layer, "mlp": {"kind": "dense", "ff": ff}}


def config(layers, width=72, vocab=130, positions=512, eps=1e-5):
    return {"architecture": "Pefisun", "width": width, "vocab": vocab, "max_positions": positions, "norm": {"eps": eps}, "layers": copy.deepcopy(layers)}


YARN = {"factor": 3.0, "original": 64, "fast": 8.0, "slow": 1.0}
MIXED = [with_mlp(lightning(), 100), with_mlp(latent(scaling=YARN), 88), with_mlp(retention(rot=8), 120), latent(heads=2, window=70), with_mlp(lightning(3, 8, 40), 56)]


class Model:
    def __init__(self, cfg, dtype, seed=0, tensors=None, max_seq_len=None):
        self.cfg, self.dtype = cfg, dtype
        self.tensors = lo.random_tensors(cfg, seed) if tensors is None else {n: lo.bf16_round(a) for n, a in tensors.items()}
        layered = pefisun.layered_config(cfg, max_seq_len, dtype == "float32")
        self.dec = rt.LayeredDecoder(layered)
        for name, layer, tensor in pefisun.tensor_names(cfg):
            bits = (np.ascontiguousarray(self.tensors[name], dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16)
            self.dec.set_tensor(layer, tensor, bits)

    def tokens(self, n, seed=1):
        return np.random.default_rng(seed).integers(0, self.cfg["vocab"], n)

    def run(self, tokens, portions=None):
        """Logits of every position, the sequence cut into `portions`."""
        self.dec.reset()
        out, at = [], 0
        for n in portions or [len(tokens)]:
            out.append(self.dec.extend(tokens[at:at + n], range(n)))
            at += n
        assert at == len(tokens) and self.dec.position == at
        return np.concatenate(out)

    def oracle(self, tokens, **kw):
        return lo.forward(self.cfg, self.tensors, tokens, **kw)

    def close(self):
        self.dec.close()


def rel(got, want):
    d = got - want
    d = d - d.mean(axis=-1, keepdims=True)
    return np.sqrt((d * d).mean(axis=-1)) / np.sqrt((want * want).mean())


def check(got, want, dtype, factor=1.0):
    e = rel(np.asarray(got, dtype=np.float64), want)
    assert np.all(np.isfinite(e)) and e.max() <= factor * TOL[dtype], (int(e.argmax()), float(e.max()))


def parts(n, sizes):
    out = []
    while sum(out) < n:
        out.append(min(sizes[len(out) % len(sizes)], n - sum(out)))
    return out


# ---- mechanisms alone ------------------------------------------------------------------------------------------------------
ALONE = {"retention": retention(), "retention_partial_rotation": retention(3, 20, 12, rot=12), "retention_no_decay": retention(1, 32, 32, decay=[1.0]),
         "retention_fast_decay": retention(2, 16, 16, decay=[0.4, 0.7]), "lightning_fast_decay": lightning(2, 16, 16, decay=[0.0, 0.05]),
         "lightning": lightning(), "lightning_one_head": lightning(1, 40, 8, decay=[0.999]),
         "latent": latent(), "latent_yarn": latent(scaling=YARN), "latent_window_1": latent(window=1), "latent_no_cut": latent(window=512),
         "latent_many_heads": latent(heads=19, dim=8, rot_dim=4, vdim=8, kv_rank=24)}


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", sorted(ALONE))
def test_mixer_alone(cuda, name, dtype):
    m = Model(config([ALONE[name]]), dtype, seed=5)
    tokens = m.tokens(90)
    want = m.oracle(tokens)
    check(m.run(tokens), want, dtype)
    check(m.run(tokens[:40], [1] * 40), want[:40], dtype)  # from the first token on, one by one
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
def test_feed_forward_norms_and_positions_alone(cuda, dtype):
    cfg = config([with_mlp(lightning(1, 8, 8), 200)], width=64, eps=3e-3)  # eps large enough to be seen
    T = lo.random_tensors(cfg, 2)
    T["l0.mix.o"] = np.zeros_like(T["l0.mix.o"])  # the mixer adds nothing
    T["l0.mlp.act"] = np.array([0.3, -0.8, 0.6, 0.4])
    T["embed"] = T["embed"] * 0.1
    m = Model(cfg, dtype, tensors=T)
    tokens = m.tokens(20)
    per = []
    want = m.oracle(tokens, per_layer=per)
    check(m.run(tokens), want, dtype)
    check(m.run(tokens, [1] * 20), want, dtype)
    m.dec.reset()
    got = m.dec.layer_residuals(tokens)
    check(got[0], per[0], dtype)
    for changed in ("pos", "l0.norm2", "final.norm"):  # each of them shows
        T2 = {**m.tensors, changed: np.zeros_like(m.tensors[changed])}
        assert rel(lo.forward(cfg, T2, tokens), want).max() > 3 * TOL["bfloat16"], changed
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
def test_residual_stream_layer_by_layer(cuda, dtype):
    m = Model(config(MIXED), dtype, seed=3)
    tokens = m.tokens(75)
    per = []
    m.oracle(tokens, per_layer=per)
    m.dec.reset()
    first = m.dec.layer_residuals(tokens[:33])
    rest = m.dec.layer_residuals(tokens[33:])
    for l, want in enumerate(per):
        check(np.concatenate([first[l], rest[l]]), want, dtype)
    m.close()


# ---- prompts, portions, decoding ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("sizes", [[200], [2], [3, 64, 1, 5], [63, 2, 65], [64], [70, 1, 1, 2], [199, 1]])
def test_cuts_do_not_matter(cuda, dtype, sizes):
    m = Model(config(MIXED), dtype, seed=7)
    tokens = m.tokens(200)
    want = m.oracle(tokens)
    check(m.run(tokens, parts(200, sizes)), want, dtype)
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
def test_long_decoding_and_first_tokens(cuda, dtype):
    m = Model(config(MIXED), dtype, seed=8)
    tokens = m.tokens(330)
    want = m.oracle(tokens)
    check(m.run(tokens, [5] + [1] * 325), want, dtype)
    for n in (1, 2, 3):
        check(m.run(tokens[:n]), want[:n], dtype)
        check(m.run(tokens[:n], [1] * n), want[:n], dtype)
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
def test_a_sequence_leaves_nothing_behind(cuda, dtype):
    m = Model(config(MIXED), dtype, seed=9)
    a, b = m.tokens(150, 2), m.tokens(37, 3)
    alone = {}
    for name, t in (("a", a), ("b", b)):
        fresh = Model(config(MIXED), dtype, tensors=m.tensors)
        alone[name] = fresh.run(t, parts(len(t), [20, 1]))
        fresh.close()
    for _ in range(2):
        np.testing.assert_array_equal(m.run(a, parts(150, [20, 1])), alone["a"])
        np.testing.assert_array_equal(m.run(b, parts(37, [20, 1])), alone["b"])
    m.close()


def test_prompt_longer_than_one_pass(cuda):
    cfg = config([with_mlp(retention(1, 16, 16), 32), latent(heads=1, window=300), lightning(1, 16, 16, decay=[0.9995])], width=32, vocab=64, positions=4600)
    m = Model(cfg, "bfloat16", seed=4)
    tokens = m.tokens(4400)
    whole = m.run(tokens)
    cut = m.run(tokens, parts(4400, [997, 64, 1]))
    check(cut, whole.astype(np.float64), "bfloat16")
    m.close()


# ---- other sizes ---------------------------------------------------------------------------------------------------------------
ODD = {"odd": (config([with_mlp(retention(3, 10, 7, rot=6), 37), with_mlp(latent(heads=5, dim=9, rot_dim=6, vdim=11, kv_rank=21, window=5), 51),
                       with_mlp(lightning(1, 13, 5), 29)], width=51, vocab=77), 140),
       "ones": (config([with_mlp(retention(1, 2, 1, rot=2), 1), with_mlp(latent(heads=1, dim=1, rot_dim=2, vdim=1, kv_rank=1, window=2), 3),
                        with_mlp(lightning(1, 1, 1), 2)], width=9, vocab=5), 70),
       "wide_heads": (config([retention(1, 200, 130, rot=64), latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=512, window=90),
                              lightning(2, 128, 72)], width=256), 150),
       "long_keys": (config([retention(1, 256, 64), lightning(1, 250, 33)], width=64), 130),
       "beyond_the_fast_forms": (config([retention(1, 300, 16, rot=300), latent(heads=2, dim=200, rot_dim=72, vdim=140, kv_rank=530, window=33)], width=64), 80)}


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", sorted(ODD))
def test_other_sizes(cuda, name, dtype):
    cfg, n = ODD[name]
    m = Model(cfg, dtype, seed=11)
    tokens = m.tokens(n)
    want = m.oracle(tokens)
    # (one-wide layers put a root mean square over a single value on everything: rounding is not averaged there)
    factor = 3.0 if name == "ones" else 1.5
    check(m.run(tokens), want, dtype, factor)
    check(m.run(tokens, parts(n, [31, 2, 1, 1])), want, dtype, factor)
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
def test_wanted_rows_with_and_without_the_last(cuda, dtype):
    """The last row's logits come from the projection that finds the next token; asked for alone, among others and not at all, in
    one portion and in portions of one row, every row is the oracle's."""
    m = Model(config([with_mlp(lightning(), 100), latent(heads=2, window=70)]), dtype, seed=4)
    tokens = m.tokens(9)
    want = m.oracle(tokens)
    session = Session(m.dec)
    for rows in ([8], [0, 8], [7], [2, 7], list(range(9))):
        session.reset_sequence()
        check(session.extend([int(t) for t in tokens], rows), want[rows], dtype, 1.5)
        check(np.asarray(session.next_logits_to_host(), dtype=np.float64).reshape(1, -1), want[8:9], dtype, 1.5)
    m.dec.reset()
    for i in range(9):
        check(m.dec.extend(tokens[i:i + 1], [0]), want[i:i + 1], dtype, 1.5)
    m.close()


@pytest.mark.parametrize("window", [1, 100, 128, 300, 512])
def test_latent_prompt_over_tiles(cuda, window):
    """Latent heads of 128 + 64 and 128 (attention on tensor memory): every position of a prompt of several 128-row blocks and 128-key
    tiles, in one portion and in portions that start and end inside both, windows that start inside a tile and that see all."""
    n = 390
    cfg = config([latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=64, window=window, scale=192 ** -0.5)], width=128, positions=512)
    m = Model(cfg, "bfloat16", seed=window)
    tokens = m.tokens(n)
    want = m.oracle(tokens)
    check(m.run(tokens), want, "bfloat16", 1.5)
    check(m.run(tokens, [127, 2, 129, 132]), want, "bfloat16", 1.5)
    check(m.run(tokens, [5, 256, 129]), want, "bfloat16", 1.5)
    m.close()


@pytest.mark.parametrize("window", [100, 512])
def test_latent_prompt_keeps_values_out_of_rows_that_do_not_attend_them(cuda, window):
    """A token whose value overflows to infinity in two columns: the rows in front of it and those whose window has left it are bit for
    bit what they are with another token in its place, those that attend it are not.  (The output projection's two columns bring values
    of about 1e34 back to the size of the residual.)"""
    n = 390
    cfg = config([latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=64, window=window, scale=192 ** -0.5)], width=128, positions=512)
    t = lo.random_tensors(cfg, 3)
    t["embed"][:, 0] = t["pos"][:, 0] = 0.0
    t["embed"][1] = 0.0
    t["embed"][1, 0] = 11.0  # an entry of its own, which latent entry 3 is made of
    t["l0.mix.dkv"][3] *= 1e-3
    t["l0.mix.dkv"][3, 0] = 4.0
    columns = [5, 255]
    t["l0.mix.uv"][columns] = 0.0
    t["l0.mix.uv"][columns, 3] = 3e38
    t["l0.mix.o"][:, columns] *= 1e-34
    m = Model(cfg, "bfloat16", tensors=t)
    tokens = np.random.default_rng(window).integers(2, cfg["vocab"], n)
    want = m.run(tokens)
    assert np.isfinite(want).all()
    for at in (5, 127, 128, 200, 289, 389):
        marked = tokens.copy()
        marked[at] = 1
        got = m.run(marked)
        seen = (np.arange(n) >= at) & (np.arange(n) < at + window)
        np.testing.assert_array_equal(got[~seen], want[~seen], err_msg=str(at))
        assert (got[seen] != want[seen]).any(axis=1).all(), at
    m.close()


# ---- one key that stands out ---------------------------------------------------------------------------------------------------
MARK, ASK = 1, 2  # token MARK leaves a key that token ASK looks for


def beacon(layer, gain, width=96, vocab=60, positions=512):
    """A one-layer model whose token MARK leaves a value that token ASK picks up: both embeddings are axes of their own, ASK's
    query points along MARK's key.  No position vectors, so the pair means the same everywhere."""
    cfg = config([layer], width=width, vocab=vocab, positions=positions)
    T = lo.random_tensors(cfg, 21)
    T["pos"][:] = 0.0
    T["l0.norm1"][:] = 0.0
    T["embed"][:, :2] = 0.0
    T["embed"][[MARK, ASK]] = 0.0
    axis = {MARK: 0, ASK: 1}
    for t, i in axis.items():
        T["embed"][t, i] = np.sqrt(width)  # after the norm: sqrt(width) along axis i
    m = layer["mixer"]
    H, d = m["heads"], m["dim"]
    e = np.sqrt(width)
    if layer["type"] == "latent_attention":
        c = lo.rms_norm_plain(T["l0.mix.dkv"][:m["kv_rank"], 0] * e, T["l0.mix.dkv.norm"], 1e-5)
        key = (T["l0.mix.uk"] @ c).reshape(H, d)
        T["l0.mix.q"][:, 1] = 0.0
        q = T["l0.mix.q"].reshape(H, d + m["rot_dim"], width)
        q[:, :d, 1] = gain * key / (e * m["scale"] * (key * key).sum(1, keepdims=True))  # score of the pair = gain
    else:
        act = lo.silu if layer["type"] == "lightning" else (lambda z: z)
        T["l0.mix.k"][:, 0] = np.abs(T["l0.mix.k"][:, 0]) * 12.0  # a strong key; positive, so that SiLU keeps it
        T["l0.mix.q"][:, 1] = gain * act(T["l0.mix.k"][:, 0] * e) / e
    return cfg, {n: lo.bf16_round(a) for n, a in T.items()}


def placed(n, marks, asks, vocab=60, seed=5):
    t = np.random.default_rng(seed).integers(3, vocab, n)
    t[list(marks)] = MARK
    t[list(asks)] = ASK
    return t


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [2, 7, 16, 64, 65, 100])
def test_window_edges(cuda, dtype, window):
    cfg, T = beacon(latent(heads=2, dim=16, rot_dim=8, vdim=24, kv_rank=40, window=window), 9.0)
    m = Model(cfg, dtype, tensors=T)
    # one query that just sees its mark, and later one that just misses its own
    p = window + 20
    n = p + window + 5
    tokens = placed(n, [p - window + 1, n - 1 - window], [p, n - 1])
    want = m.oracle(tokens)
    for w in (window - 1, window + 1):  # an edge that is one token off shows in the logits
        off = copy.deepcopy(cfg)
        off["layers"][0]["mixer"]["mask"]["size"] = w
        assert rel(lo.forward(off, m.tensors, tokens), want).max() > 5 * TOL["bfloat16"], w
    check(m.run(tokens), want, dtype)                                        # in a prompt
    check(m.run(tokens, [p] + [1] * (n - p)), want, dtype)                   # decoded
    check(m.run(tokens, [p - 1] + parts(n - p + 1, [2, 3])), want, dtype)    # in short portions
    check(m.run(tokens, [p - window + 2, n - p - 5, window - 3 + 6] if window > 2 else [p, 2, n - p - 2]), want, dtype)  # the mark ends a portion
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kind", ["retention", "lightning"])
def test_far_keys_and_chunk_edges(cuda, dtype, kind):
    decay = [0.9999, 0.98]
    layer = retention(2, 16, 24, decay=decay, rot=2, base=1e9) if kind == "retention" else lightning(2, 24, 16, decay=decay)
    cfg, T = beacon(layer, 2.0)
    m = Model(cfg, dtype, tensors=T)
    for distance in (1, 63, 64, 65, 127, 128, 129, 300):
        n = distance + 6
        tokens = placed(n, [4], [4 + distance])
        want = m.oracle(tokens)
        without = tokens.copy()
        without[4] = 9
        assert rel(m.oracle(without), want)[4 + distance] > 5 * TOL["bfloat16"], distance  # the mark is seen from there
        check(m.run(tokens), want, dtype)
        check(m.run(tokens, [distance + 3, 1, 1, 1]), want, dtype)
        check(m.run(tokens, [5, distance + 1]), want, dtype)      # the mark ends a portion
        check(m.run(tokens, [4] + parts(distance + 2, [64, 2])), want, dtype)
    m.close()


@pytest.mark.parametrize("dtype", DTYPES)
def test_decay_of_every_head_counts(cuda, dtype):
    layer = lightning(3, 16, 16, decay=[0.5, 0.9, 0.99])
    cfg = config([layer])
    m = Model(cfg, dtype, seed=6)
    tokens = m.tokens(100)
    want = m.oracle(tokens)
    check(m.run(tokens), want, dtype)
    check(m.run(tokens, [60] + [1] * 40), want, dtype)
    swapped = copy.deepcopy(cfg)
    swapped["layers"][0]["mixer"]["decay"] = [0.9, 0.5, 0.99]
    assert rel(lo.forward(swapped, m.tensors, tokens), want).max() > 3 * TOL["bfloat16"]
    m.close()


def test_plain_forms_agree_with_the_fast_ones(cuda, monkeypatch):
    monkeypatch.setenv("KMLL_LAYERED", "plain")
    plain = Model(config(MIXED), "bfloat16", seed=12)
    monkeypatch.delenv("KMLL_LAYERED")
    fast = Model(config(MIXED), "bfloat16", tensors=plain.tensors)
    tokens = plain.tokens(130)
    want = plain.oracle(tokens)
    for cut in ([130], [100] + [1] * 30):
        check(plain.run(tokens, cut), want, "bfloat16")
        check(fast.run(tokens, cut), want, "bfloat16")
    plain.close()
    fast.close()


# ---- generation through the session layer -----------------------------------------------------------------------------------
@pytest.fixture
def model_dir(tmp_path):
    cfg = config(MIXED)
    T = lo.random_tensors(cfg, 14)
    (tmp_path / "config.json").write_text(json.dumps(cfg))
    write_safetensors(str(tmp_path / "model.safetensors"), {n: (np.ascontiguousarray(a).view(np.uint32) >> 16).astype(np.uint16) for n, a in T.items()})
    return str(tmp_path), cfg, T


@pytest.mark.parametrize("dtype", DTYPES)
def test_greedy_generation(cuda, model_dir, dtype):
    path, cfg, T = model_dir
    s = Session(registry.load_model(path, dtype, max_seq_len=160))
    prompt = np.random.default_rng(6).integers(0, cfg["vocab"], 45)
    res = s.run_generation_request(prompt, GenerationOptions(max_new_tokens=40))
    gen = res["generated_tokens"]
    assert len(gen) == 40 and res["finish_reason"] == ("max-new-tokens", None) and res["backend"].startswith("bf16")
    mem = res["memory_stats"]
    assert mem["weights_bytes"] > 0 and mem["kv_cache_bytes"] > 0
    # the oracle, fed the same tokens, prefers each of them (within its tolerance where two are close)
    want = lo.forward(cfg, T, np.concatenate([prompt, gen]))
    scale = np.sqrt((want * want).mean())
    for i, t in enumerate(gen):
        row = want[len(prompt) + i - 1]
        assert row.max() - row[t] <= 6 * TOL[dtype] * scale, i
    # a stop token ends the run whatever the size of the device-resident chunks, and the sequence goes on from there
    stop = gen[17]
    first = gen.index(stop)
    for chunk in (16, 7, 1):
        s.CHUNK = chunk
        s.prefill(prompt)
        steps = s.generate_greedy_until(40, 1, stop)
        assert [x.token_id for x in steps] == gen[:first + 1]
        more = s.generate_greedy_until(5)
        assert [x.token_id for x in more] == gen[first + 1:first + 6]
    # the k-best loop and cold sampling take the same tokens; the logits are those of the decode steps
    s.prefill(prompt)
    assert [x.token_id for x in s.generate_greedy_until(8, 3)] == gen[:8]
    s.prefill(prompt)
    assert [x.token_id for x in s.generate_sampled_top_k_until(8, 4, None, SamplingOptions(temperature=0.0))] == gen[:8]
    logits = s.next_logits_to_host()
    assert rel(logits[None].astype(np.float64), want[len(prompt) + 7][None]).max() <= 2 * TOL[dtype]
    # a prompt in portions generates the same
    s.reset_sequence()
    s.extend(prompt[:20])
    s.extend(prompt[20:])
    assert [x.token_id for x in s.generate_greedy_until(10)] == gen[:10]
    with pytest.raises(KmllError):
        s.run_generation_request(prompt, GenerationOptions(max_new_tokens=200))
    s.dec.close()


def test_rewind_replays_the_states(cuda):
    m = Model(config(MIXED), "float32", seed=15, max_seq_len=200)
    tokens = m.tokens(60)
    m.dec.prefill(tokens)
    toks, _ = m.dec.generate_greedy(20)
    seq = np.concatenate([tokens, toks])
    want = m.oracle(seq)
    for position in (75, 60, 33):  # behind the remembered state, at it, ahead of it (the whole prompt is replayed)
        m.dec.rewind(position)
        assert m.dec.position == position
        check(m.dec.extend(seq[position:position + 5], range(5)), want[position:position + 5], "float32")
        m.dec.prefill(tokens)
        m.dec.generate_greedy(20)
    h, _ = m.dec.history(0, 20)
    assert list(h) == list(toks)
    m.close()


def test_limits_are_errors(cuda):
    m = Model(config([lightning()], positions=40), "bfloat16")
    with pytest.raises(KmllError):
        m.dec.extend(m.tokens(41))
    with pytest.raises(KmllError):
        m.dec.extend([m.cfg["vocab"]])
    with pytest.raises(KmllError):
        m.dec.extend([1, 2], [1, 0])
    with pytest.raises(KmllError):
        rt.BatchDecoder(m.dec, 2)
    with pytest.raises(KmllError):
        m.dec.prefill(m.tokens(5), token_loop=True)
    m.dec.reset()
    assert m.dec.extend(m.tokens(40), [39]).shape == (1, m.cfg["vocab"])
    with pytest.raises(KmllError):
        m.dec.extend([1])
    missing = rt.LayeredDecoder(pefisun.layered_config(m.cfg))
    with pytest.raises(KmllError):
        missing.extend([1])  # no weights
    with pytest.raises(KmllError):
        missing.set_tensor(0, rt.T_UK, np.zeros((1, 1), np.uint16))
    assert load().kmll_decoder_init_random(missing._h, 3, 0.05, 1) == 0
    assert np.isfinite(missing.extend(m.tokens(20), [19])).all()
    back = m.dec.get_tensor(0, rt.T_WQ)
    np.testing.assert_array_equal(back, (m.tensors["l0.mix.q"].view(np.uint32) >> 16).astype(np.uint16))
    missing.close()
    m.close()


def test_uniform_decoder_extends_by_decode_steps(cuda):
    cfg = rt.DecoderConfig(dim=256, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=64, hidden_dim=512, vocab_size=640, max_seq_len=64, format=rt.FORMAT_RS_I8)
    dec = rt.Decoder(cfg)
    dec.init_random(3, 0.05)
    t = np.random.default_rng(1).integers(0, 640, 12)
    s = Session(dec)
    got = s.extend(t[:7], [6])
    got2 = s.extend(t[7:], [0, 4])
    ref = Session(dec)
    for n, row in ((7, got[0]), (8, got2[0]), (12, got2[1])):
        ref.prefill(t[:n])
        np.testing.assert_allclose(row, ref.next_logits_to_host(), atol=2e-3)
    dec.close()


# ---- operators through the C ABI --------------------------------------------------------------------------------------------
def test_bf16_linear_operators(cuda):
    import torch

    from kmll_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(9)

    def randn(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    ws = ops.linear_batched_bf16_workspace()
    for batch, rows, cols in ((1, 5, 8), (3, 130, 72), (17, 200, 520), (40, 1000, 2056), (64, 128, 4096), (256, 384, 1024), (300, 1300, 320), (700, 96, 64)):
        w = (randn(rows, cols) / cols ** 0.5).bfloat16()
        x, res = randn(batch, cols), randn(batch, rows)
        want = x.bfloat16().double() @ w.double().T + res.double()
        for workspace in (None, ws, ws):
            got = ops.linear_batched_bf16(x.bfloat16(), w, residual=res, workspace=workspace)
            assert float((got.double() - want).abs().max()) <= 2e-5 * cols ** 0.5, (batch, rows, cols)
        got = ops.linear_batched_bf16(x.bfloat16(), w, out_bf16=True, workspace=ws)
        assert float((got.double() - (want - res.double())).abs().max()) <= 0.03
        want = x.double() @ w.double().T + res.double()
        assert float((ops.linear_batched_bf16(x, w, residual=res).double() - want).abs().max()) <= 1e-5 * cols ** 0.5
        norm = randn(cols).bfloat16()
        xd, w0 = x[0].double(), w.double()
        got = ops.linear_bf16(x[0].contiguous(), w, residual=res[0].contiguous())
        assert float((got.double() - (w0 @ xd + res[0].double())).abs().max()) <= 1e-5 * cols ** 0.5
        n = torch.from_numpy(lo.rms_norm_zero_centred(xd.cpu().numpy(), norm.double().cpu().numpy(), 1e-3)).cuda()
        y = w0 @ n
        y[:rows // 2] = y[:rows // 2] * torch.sigmoid(y[:rows // 2])
        got = ops.linear_bf16(x[0].contiguous(), w, norm_weight=norm, norm_offset=1.0, eps=1e-3, silu_rows=rows // 2)
        assert float((got.double() - y).abs().max()) <= 4e-5 * cols ** 0.5
        coef = randn(4).bfloat16()
        n = torch.from_numpy(lo.poly_norm(xd.cpu().numpy(), coef.double().cpu().numpy(), 1e-3)).cuda()
        got = ops.polynorm_linear_bf16(x[0].contiguous(), coef, 1e-3, w)
        assert float((got.double() - w0 @ n).abs().max()) <= 6e-5 * cols ** 0.5
        gate = randn(cols)
        o = xd.cpu().numpy()
        n = lo.rms(o.reshape(-1, 8), 1e-3).reshape(-1) * lo.silu(gate.double().cpu().numpy())
        got = ops.gated_linear_bf16(x[0].contiguous(), gate, w, 1e-3, head_len=8)
        assert float((got.double() - w0 @ torch.from_numpy(n).cuda()).abs().max()) <= 4e-5 * cols ** 0.5
        n = lo.rms_norm_plain(o, norm.double().cpu().numpy(), 1e-3) * lo.sigmoid(gate.double().cpu().numpy())
        got = ops.gated_linear_bf16(x[0].contiguous(), gate, w, 1e-3, norm_weight=norm, sigmoid=True)
        assert float((got.double() - w0 @ torch.from_numpy(n).cuda()).abs().max()) <= 4e-5 * cols ** 0.5


def test_norm_weights_of_the_launch_in_front(cuda):
    """Norm weights that the launch directly in front writes - a long one, which ends with them - are the ones that the projection
    uses, in every form that loads them in whole pieces.  Bounds as in test_operators_against_64_bits."""
    import torch

    from kmll_b200 import ops

    cols, rows, eps = 2048, 160, 1e-3
    gen = torch.Generator(device="cuda").manual_seed(21)
    w = (torch.randn(rows, cols, generator=gen, device="cuda") / cols ** 0.5).bfloat16()
    x, gate = (torch.randn(cols, generator=gen, device="cuda") for _ in range(2))
    xd, gd, w0 = x.double(), gate.double(), w.double()
    source = torch.zeros(1 << 25, device="cuda")
    linear = rt.MixerSpec(rt.MIXER_GATED_LINEAR, cols // 128, 128, 128, out_norm=rt.OUT_NORM_HEAD_WEIGHTED, gate_act=rt.ACT_SILU)
    centred = xd - xd.mean()
    normed = xd / (xd.square().mean() + eps).sqrt()
    by_head = (xd.view(-1, 128) / (xd.view(-1, 128).square().mean(1, keepdim=True) + eps).sqrt()).reshape(-1)
    silu = gd * torch.sigmoid(gd)
    forms = [(lambda n: ops.linear_bf16(x, w, norm_weight=n, eps=eps), lambda n: normed * n),
             (lambda n: ops.normed_linear_bf16(x, w, rt.NORM_LAYER, n, n, eps), lambda n: centred / (centred.square().mean() + eps).sqrt() * n + n),
             (lambda n: ops.gated_linear_bf16(x, gate, w, eps, norm_weight=n), lambda n: normed * n * silu),
             (lambda n: ops.mixer_output_linear_bf16([linear], x, [n[:128]], [gate], w, eps), lambda n: by_head * n[:128].repeat(cols // 128) * silu)]
    for i in range(12):
        source[-cols:] = torch.randn(cols, generator=gen, device="cuda") + 1.0
        for call, value in forms:
            got = call(ops.f32_to_bf16(source)[-cols:])
            want = w0 @ value(source[-cols:].bfloat16().double())
            assert float((got.double() - want).abs().max()) <= 4e-5 * cols ** 0.5, i
    # written long before: the same values
    n = ops.f32_to_bf16(source)[-cols:]
    torch.cuda.synchronize()
    for call, value in forms:
        assert float((call(n).double() - w0 @ value(n.double())).abs().max()) <= 4e-5 * cols ** 0.5


@pytest.mark.parametrize("cols", [256, 384, 4096, 4224, 8192, 8320])
def test_mixer_output_of_whole_heads(cuda, cols):
    """The output projection of mixers whose heads are runs of 128 columns (all of x in whole pieces), of 8192 columns, of more and with
    heads of 256 (one column at a time): every norm, gates by column and by head, one and two mixers, x on and off a 16-byte
    boundary.  Bound: f32 sums of `cols` products around 1, as in test_bf16_linear_operators."""
    import torch

    from kmll_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(cols)
    eps, rows = 1e-3, 70
    w = (torch.randn(rows, cols, generator=gen, device="cuda") / cols ** 0.5).bfloat16()
    res = torch.randn(rows, generator=gen, device="cuda")
    act = {rt.ACT_SILU: torch.nn.functional.silu, rt.ACT_SIGMOID: torch.sigmoid}

    def attention(heads, vdim):
        return rt.MixerSpec(rt.MIXER_ATTENTION, heads, 64, vdim, gate_act=rt.ACT_SIGMOID, out_scale=0.6)

    def linear(heads, norm, vdim=128):
        return rt.MixerSpec(rt.MIXER_GATED_LINEAR, heads, 64, vdim, gate_act=rt.ACT_SILU, out_scale=1.3, out_norm=norm)

    norms = (rt.OUT_NORM_PER_HEAD, rt.OUT_NORM_JOINT, rt.OUT_NORM_HEAD_WEIGHTED, rt.OUT_NORM_NONE)
    n = cols // 128
    cases = [[linear(n, norm)] for norm in norms] + [[attention(n, 128)]]
    cases += [[attention(1, 128), linear(n - 1, norm)] for norm in norms] + [[linear(n - 1, norm), attention(1, 128)] for norm in norms]
    cases += [[linear(1, a), linear(n - 1, b)] for a in norms for b in norms]
    if n % 2 == 0:
        cases += [[linear(n // 2, norm, 256)] for norm in norms] + [[attention(n // 2, 256)]]
        if n > 2:
            cases += [[attention(1, 256), linear(n - 2, norm)] for norm in norms]
    for case, mixers in enumerate(cases):
        x = torch.randn(cols + 1, generator=gen, device="cuda")
        x = x[1:] if case % 4 == 3 else x[:cols]
        weights, gates, parts, at = [], [], [], 0
        for m in mixers:
            o = x[at:at + m.heads * m.vdim].double().view(m.heads, m.vdim)
            at += m.heads * m.vdim
            whole = m.mixer == rt.MIXER_ATTENTION
            norm = rt.OUT_NORM_NONE if whole else m.out_norm
            gates.append(torch.randn(m.heads if whole else m.heads * m.vdim, generator=gen, device="cuda"))
            weight = None
            if norm in (rt.OUT_NORM_JOINT, rt.OUT_NORM_HEAD_WEIGHTED):
                weight = (torch.randn(m.vdim * (m.heads if norm == rt.OUT_NORM_JOINT else 1), generator=gen, device="cuda") + 1.0).bfloat16()
            weights.append(weight)
            if norm == rt.OUT_NORM_JOINT:
                o = o / (o.square().mean() + eps).sqrt() * weight.double().view(m.heads, m.vdim)
            elif norm != rt.OUT_NORM_NONE:
                o = o / (o.square().mean(1, keepdim=True) + eps).sqrt()
                if weight is not None:
                    o = o * weight.double()
            parts.append((o * act[m.gate_act](gates[-1].double()).view(m.heads, -1) * m.out_scale).reshape(-1))
        got = ops.mixer_output_linear_bf16(mixers, x, weights, gates, w, eps, residual=res)
        want = w.double() @ torch.cat(parts) + res.double()
        assert float((got.double() - want).abs().max()) <= 4e-5 * cols ** 0.5, (case, mixers)


@pytest.mark.parametrize("cols", [4096, 4104, 8200])
def test_norm_of_long_and_unaligned_rows(cuda, cols):
    """Norms over what a thread can hold in whole pieces (4096 columns), over more, and of an x that is off a 16-byte boundary."""
    import torch

    from kmll_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(cols)
    w = (torch.randn(50, cols, generator=gen, device="cuda") / cols ** 0.5).bfloat16()
    nw, nb = (torch.randn(cols, generator=gen, device="cuda").bfloat16() for _ in range(2))
    coef = torch.randn(4, generator=gen, device="cuda").bfloat16()
    for off in (0, 1):
        x = (torch.randn(cols + 1, generator=gen, device="cuda") * 2 + 0.5)[off:off + cols]
        X = x.double()
        for got, n in ((ops.linear_bf16(x, w, norm_weight=nw, norm_offset=1.0, eps=1e-3), lo.rms_norm_zero_centred(X.cpu().numpy(), nw.double().cpu().numpy(), 1e-3)),
                       (ops.normed_linear_bf16(x, w, rt.NORM_LAYER, nw, nb, 1e-3),
                        ((X - X.mean()) / (X.var(unbiased=False) + 1e-3).sqrt() * nw.double() + nb.double()).cpu().numpy()),
                       (ops.polynorm_linear_bf16(x, coef, 1e-3, w), lo.poly_norm(X.cpu().numpy(), coef.double().cpu().numpy(), 1e-3))):
            assert float((got.double() - w.double() @ torch.from_numpy(n).cuda()).abs().max()) <= 6e-5 * cols ** 0.5, off


@pytest.mark.parametrize("tokens,position,window", [(1, 0, 0), (130, 0, 0), (300, 0, 1000), (257, 130, 0), (390, 250, 300), (128, 900, 200), (5, 700, 129)])
def test_latent_prompt_operator_with_growing_scores(cuda, tokens, position, window):
    """Latent attention of a prompt against 64-bit sums over the same bf16 operands.  Keys of the later tiles are longer, so row maxima grow
    by many powers of two from tile to tile, in some rows more than in others; a last case in each head has keys that shrink instead.
    Bound: a score is a sum of exact products in f32, 12 steps of 16 columns that each lose 2^-23 of the sum of magnitudes, and its weight
    follows it; a weight is two bf16 planes (2^-16).  Both enter sum and divisor, hence the two."""
    import torch

    from kmll_b200 import ops

    heads, dim, rot, vdim, rank, max_seq = 3, 128, 64, 128, 64, 1100
    gen = torch.Generator(device="cuda").manual_seed(tokens + window)
    seen = position + tokens
    first = max(0, position - window + 1) if window else 0
    length = torch.linspace(0.2, 6.0, seen, device="cuda")
    k = torch.randn(seen, heads, dim, generator=gen, device="cuda") * torch.stack([length, length, length.flip(0)], 1)[:, :, None]
    v = torch.randn(seen, heads, vdim, generator=gen, device="cuda")
    expanded = torch.cat([k.reshape(seen, -1), v.reshape(seen, -1)], 1).bfloat16()[first:].contiguous()
    cache = torch.zeros(max_seq, rank + rot, device="cuda", dtype=torch.bfloat16)
    cache[:seen, rank:] = torch.randn(seen, rot, generator=gen, device="cuda").bfloat16()
    angle = torch.rand(max_seq, rot // 2, generator=gen, device="cuda") * 6.28
    turn = (torch.stack([angle.cos(), angle.sin()], 2) * 16).round().contiguous() / 16  # (rotated entries are exact in f32, whatever the order)
    x = torch.randn(tokens, heads * (dim + rot) + 8, generator=gen, device="cuda").bfloat16()
    scale = 192 ** -0.5 * 1.7
    out = ops.latent_attention_prefill(x, position, heads, dim, rot, vdim, rank, window, scale, turn, cache, expanded, first).double()
    q = x[:, :heads * (dim + rot)].float().view(tokens, heads, dim + rot)
    c, s = (turn[position:seen, None, :, i] for i in range(2))
    u, z = q[:, :, dim:dim + rot // 2], q[:, :, dim + rot // 2:]
    q = torch.cat([q[:, :, :dim], u * c - z * s, z * c + u * s], 2).bfloat16().double()
    both = expanded.double()
    K, V = both[:, :heads * dim].view(-1, heads, dim), both[:, heads * dim:].view(-1, heads, vdim)
    K = torch.cat([K, cache[first:seen, None, rank:].double().expand(-1, heads, -1)], 2)
    scores = torch.einsum("thd,shd->hts", q, K) * scale
    at, of = torch.arange(position, seen, device="cuda")[:, None], torch.arange(first, seen, device="cuda")[None]
    hidden = (of > at) | (of <= at - window if window else torch.zeros_like(of, dtype=torch.bool))
    weights = torch.softmax(scores.masked_fill(hidden, float("-inf")), 2)
    want = torch.einsum("hts,shd->thd", weights, V)
    spread = torch.einsum("hts,shd->thd", weights, V.abs())
    size = torch.einsum("thd,shd->hts", q.abs(), K.abs()) * scale
    slack = (size.masked_fill(hidden, 0.0).amax(2) * 12 * 2.0 ** -23 + 2.0 ** -16).T[:, :, None]
    rel = ((out.view(tokens, heads, vdim) - want).abs() / (spread * slack * 2)).amax()
    assert float(rel) <= 1.0, float(rel)


# more than 256 rows of x: pairs of blocks.  One k-tile (one accumulator), a ragged last one, one row of weights, ragged tiles on both
# sides, several units per pair
@pytest.mark.parametrize("tokens,rows,cols", [(257, 130, 72), (300, 2, 64), (513, 520, 200), (640, 257, 1000), (1030, 6000, 136), (2500, 384, 4104)])
def test_bf16_gemm_of_many_rows(cuda, tokens, rows, cols):
    """Against 64-bit sums: f32 accumulation in steps of 16 columns (2^-23 of the partial sum each), bf16 results half an ulp more."""
    import torch

    from kmll_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, cols, generator=gen, device="cuda").bfloat16()
    w = torch.randn(rows, cols, generator=gen, device="cuda").bfloat16()
    res = torch.randn(tokens, rows, generator=gen, device="cuda")
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = (cols / 16 + 8) * 2.0 ** -23 * (size + res.double().abs())
    assert bool(((ops.linear_batched_bf16(x, w, residual=res).double() - want - res.double()).abs() <= bound).all())
    assert bool(((ops.linear_batched_bf16(x, w, out_bf16=True).double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all())
    if rows % 2 == 0:
        gate, up = want[:, 0::2], want[:, 1::2]
        got = ops.pair_linear_batched_bf16(x, w, 1).double()  # SiLU
        pair = torch.nn.functional.silu(gate) * up
        slack = bound[:, 0::2] * up.abs() * 1.1 + bound[:, 1::2] * gate.abs() + 2.0 ** -20 * pair.abs()
        assert bool(((got - pair).abs() <= slack + 2.0 ** -8 * pair.abs()).all())
