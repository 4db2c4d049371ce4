"""GPU parity tests of the decode runtime against the CPU oracle model: same quantized bytes on both
sides, identical greedy tokens (checked against the oracle's top-2 margin), logits and hidden states
within kmll's tolerances."""
import numpy as np
import pytest
import torch

from kmll_b200 import runtime as rt
from kmll_b200.lib import KmllError
from oracle_model import OracleDecoder

pytestmark = pytest.mark.gpu
F = np.float32


def tiny(fmt, fused=True, **kw):
    base = dict(n_layers=2, dim=256, n_heads=4, n_kv_heads=2, head_dim=64, hidden_dim=512, vocab_size=640, rope_theta=1e6, norm_eps=1e-6,
                max_seq_len=48, format=fmt, fused=fused)
    base.update(kw)
    return rt.DecoderConfig(**base)


def make(cfg, seed=2, std=0.05, tie=False):
    dec = rt.Decoder(cfg)
    dec.init_random(seed, std, tie)
    return dec


def check_against_oracle(dec, cfg, prompt, n_steps, batched_prefill, hid_tol=2e-4, min_margin=1e-3, logit_tol=1e-3):
    ora = OracleDecoder(cfg, dec)
    logits = ora.prefill(prompt)
    dec.prefill(prompt, token_loop=not batched_prefill)
    hid = dec.last_hidden()
    scale = np.max(np.abs(ora.hidden))
    assert np.max(np.abs(hid - ora.hidden)) <= hid_tol * max(scale, 1.0), "hidden state after prefill"
    steps, _ = ora.generate_greedy(logits, n_steps)
    tokens, glogits = dec.generate_greedy(n_steps)
    for i, (tok, logit, margin) in enumerate(steps):
        if margin < min_margin:
            break  # a near-tie in the oracle: either token is a faithful arg-max, later steps diverge legitimately
        assert int(tokens[i]) == tok, f"greedy token differs at step {i} (oracle margin {margin})"
        assert abs(float(glogits[i]) - logit) <= logit_tol * max(abs(logit), 1.0)
    assert dec.position == len(prompt) + n_steps


@pytest.mark.parametrize("fmt", [rt.FORMAT_RS_I8, rt.FORMAT_W4G128])
@pytest.mark.parametrize("fused", [True, False])
def test_decode_matches_oracle(cuda, fmt, fused):
    cfg = tiny(fmt, fused)
    dec = make(cfg)
    rng = np.random.default_rng(2)
    prompt = rng.integers(0, cfg.vocab_size, 9)
    check_against_oracle(dec, cfg, prompt, 6, batched_prefill=False)
    dec.close()


@pytest.mark.parametrize("fmt", [rt.FORMAT_RS_I8, rt.FORMAT_W4G128])
@pytest.mark.parametrize("window", [1, 24, 70])
@pytest.mark.parametrize("batched_prefill", [False, True])
def test_sliding_window_matches_oracle(cuda, fmt, window, batched_prefill):
    """sliding_window: the oracle attends the last `window` rows of its cache.  max_seq_len 200 gives the decode kernel
    four 52-position slices; with 110-token prompts a window of 24 lies inside one slice or straddles two, one of 70
    covers slices partly, and the slices before the window leave without a partial.  f32 cache: the f32 tolerances."""
    cfg = tiny(fmt, True, n_heads=8, n_kv_heads=2, head_dim=128, dim=256, max_seq_len=200, sliding_window=window)
    dec = make(cfg)
    prompt = np.random.default_rng(window).integers(0, cfg.vocab_size, 110)
    check_against_oracle(dec, cfg, prompt, 8, batched_prefill=batched_prefill)
    dec.close()


def test_sliding_window_other_step_forms_and_bf16(cuda):
    for fused, rotary_dim, kv_bf16 in [(False, None, False), (True, 32, False), (True, None, True)]:
        cfg = tiny(rt.FORMAT_W4G128, fused, rotary_dim=rotary_dim, max_seq_len=96, sliding_window=20, kv_bf16=kv_bf16)
        dec = make(cfg)
        prompt = np.random.default_rng(6).integers(0, cfg.vocab_size, 66)
        check_against_oracle(dec, cfg, prompt, 5, batched_prefill=fused, **(BF16_KV_BOUND if kv_bf16 else {}))
        dec.close()


# fused = 0 keeps the f32 prompt attention: two, four and eight query rows per thread (by heads x rows), both head sizes and cache types; windows
# that leave out whole 64-key tiles, begin inside one, hold one position, and none
@pytest.mark.parametrize("n,heads,kv,hd", [(150, 4, 2, 64), (150, 4, 1, 128), (190, 32, 8, 64), (160, 32, 4, 128), (640, 32, 8, 64), (590, 32, 8, 128)])
@pytest.mark.parametrize("window,kv_bf16", [(0, True), (1, False), (20, True), (70, False)])
def test_f32_prompt_attention_matches_oracle(cuda, n, heads, kv, hd, window, kv_bf16):
    """The last row of prompts that end at several places of a row block and of a tile, against the oracle's pass over the longest."""
    cfg = tiny(rt.FORMAT_RS_I8, False, n_layers=1, n_heads=heads, n_kv_heads=kv, head_dim=hd, max_seq_len=n + 8, sliding_window=window, kv_bf16=kv_bf16)
    dec = make(cfg)
    ora = OracleDecoder(cfg, dec)
    prompt = np.random.default_rng(n + window).integers(0, cfg.vocab_size, n)
    ends = {n, n - 1, n - 9, n - 30, n // 64 * 64, n // 64 * 64 + 1}
    for at, token in enumerate(prompt, 1):
        ora.forward(int(token))
        if at in ends:
            dec.prefill(prompt[:at])
            got = dec.last_hidden()
            scale = max(float(np.max(np.abs(ora.hidden))), 1.0)
            assert np.max(np.abs(got - ora.hidden)) <= (BF16_KV_BOUND["hid_tol"] if kv_bf16 else 2e-4) * scale, at
    dec.close()


@pytest.mark.parametrize("heads,kv,hd", [(4, 2, 64), (4, 1, 128), (8, 8, 128)])
@pytest.mark.parametrize("window,kv_bf16", [(0, False), (0, True), (1, False), (66, False), (100, True), (130, False), (300, False)])
def test_prompt_attention_tiles_match_oracle(cuda, heads, kv, hd, window, kv_bf16):
    """Attention on tensor memory: prompts that end around the 128 rows of a block and the 128 keys of a tile, one to four tiles (one and
    two streams of tiles), windows that start inside a tile; the other kernel on the other side of its lines (length, window), and for
    (8, 8, 128) with an f32 cache: keys wider than the feed-forward leave no room for planes.  Bounds as in the tests above."""
    n = 390
    cfg = tiny(rt.FORMAT_RS_I8, True, n_layers=1, n_heads=heads, n_kv_heads=kv, head_dim=hd, max_seq_len=n + 8, sliding_window=window, kv_bf16=kv_bf16)
    dec = make(cfg)
    ora = OracleDecoder(cfg, dec)
    prompt = np.random.default_rng(heads + hd + window).integers(0, cfg.vocab_size, n)
    for at, token in enumerate(prompt, 1):
        ora.forward(int(token))
        if at in (1, 2, 64, 127, 128, 129, 192, 193, 255, 256, 257, 383, 384, 385, 390):
            dec.prefill(prompt[:at])
            got = dec.last_hidden()
            scale = max(float(np.max(np.abs(ora.hidden))), 1.0)
            assert np.max(np.abs(got - ora.hidden)) <= (BF16_KV_BOUND["hid_tol"] if kv_bf16 else 2e-4) * scale, at
    dec.close()


# strength (by MARK token) of the mark in each key tile, 0: none.  Each stream of tiles (even, odd) sees its maximum grow late, early, in every
# tile, not at all; equal marks in one stream and in both
PEAKS = [(0, 0, 0, 0, 1), (0, 0, 0, 1, 0), (4, 3, 2, 1, 0), (1, 2, 3, 4, 0), (0, 1, 1, 0, 0), (1, 0, 0, 0, 1), (4, 0, 2, 0, 1), (0, 4, 0, 2, 1), (4, 4, 3, 3, 3)]


@pytest.mark.parametrize("heads,kv,hd", [(4, 2, 64), (4, 1, 128)])
@pytest.mark.parametrize("kv_bf16", [False, True])
def test_prompt_attention_with_keys_that_stand_out(cuda, heads, kv, hd, kv_bf16):
    """Scores of token ASK's query with the keys of MARK tokens are 60, 30, 15 and 7.5 (85, 42, 21 and 10 powers of two), of everything
    else about 0: the running maximum grows by more than 2^8 in the tiles that PEAKS says, in the rows that ask and not in the others
    of their warps, and the two streams meet with maxima far apart.  The scores come from one pair of entries that the rotation
    turns by 5e-4 at most; rounding of q and k moves them by 60 * 2^-16, so weights and attention by 1e-3 of themselves, a tenth of that of
    the hidden state (a mark's value is a tenth of it at most): the bounds of the tests above."""
    n, ask, pair = 640, 5, hd // 2 - 1
    cfg = tiny(rt.FORMAT_RS_I8, True, n_layers=1, n_heads=heads, n_kv_heads=kv, head_dim=hd, max_seq_len=n + 8, kv_bf16=kv_bf16)
    dec = make(cfg)
    rng = np.random.default_rng(hd + kv_bf16)
    table = (rng.normal(0, 1, (cfg.vocab_size, cfg.dim)).astype(F).view(np.uint32) >> 16).astype(np.uint16)
    table[:, 1:6] = 0
    table[1:6] = 0
    table[np.arange(1, 6), np.arange(1, 6)] = 0x4180  # 16: the norm leaves the whole row in this entry
    dec.set_tensor(-1, rt.T_EMBEDDING, table)
    dec.set_tensor(0, rt.T_ATTENTION_NORM, np.full(cfg.dim, 0x3f80, dtype=np.uint16))
    for tensor, count in ((rt.T_WQ, heads), (rt.T_WK, kv)):
        values, scales = dec.get_tensor(0, tensor)
        for h in range(count):
            rows = [h * hd + pair, h * hd + hd - 1]
            values[rows] = 0
            if tensor == rt.T_WQ:
                values[rows[0], ask] = 127
            else:
                values[rows[0], 1:5] = (127, 64, 32, 16)
            scales[rows] = (60 * hd ** 0.5) ** 0.5 / (127 * 16)
        dec.set_tensor(0, tensor, values, scales)
    for peaks in PEAKS:
        prompt = rng.integers(6, cfg.vocab_size, n)
        prompt[rng.random(n) < 0.3] = ask
        for tile, mark in enumerate(peaks):
            if mark:
                prompt[tile * 128 + int(rng.integers(3, 120))] = mark
        ora = OracleDecoder(cfg, dec)
        ends = {257, 300, 384, 385, 500, 512, 513, 600, 638, 640}
        for at, token in enumerate(prompt, 1):
            if at in ends:
                token = prompt[at - 1] = ask if at != 638 else 7
            ora.forward(int(token))
            if at in ends:
                dec.prefill(prompt[:at])
                scale = max(float(np.max(np.abs(ora.hidden))), 1.0)
                worst = float(np.max(np.abs(dec.last_hidden() - ora.hidden))) / scale
                assert worst <= (BF16_KV_BOUND["hid_tol"] if kv_bf16 else 2e-4), (peaks, at, worst)
    dec.close()


@pytest.mark.parametrize("heads,kv,hd,kv_bf16,window", [(4, 2, 64, False, 260), (4, 2, 64, True, 520), (4, 1, 128, False, 100), (4, 1, 128, True, 100)])
def test_prompt_attention_keeps_values_out_of_rows_that_do_not_attend_them(cuda, heads, kv, hd, kv_bf16, window):
    """Token MARK's value overflows to infinity in two columns of a head.  Just in front of the last row's window, in a tile that
    rows of its block do attend, the last row is bit for bit what it is with another token there; inside the window it is not.
    The output projection's scales bring the two columns, about 1e36, back to the size of the residual."""
    mark, columns, whole = 1, [5, hd - 1], (window // 128 + 3) * 128
    cfg = tiny(rt.FORMAT_RS_I8, True, n_layers=1, n_heads=heads, n_kv_heads=kv, head_dim=hd, max_seq_len=whole + 8, sliding_window=window, kv_bf16=kv_bf16)
    dec = make(cfg)
    rng = np.random.default_rng(hd)
    table = (rng.normal(0, 1, (cfg.vocab_size, cfg.dim)).astype(F).view(np.uint32) >> 16).astype(np.uint16)
    table[:, 0] = 0
    table[mark] = 0
    table[mark, 0] = 0x4180  # 16: the norm leaves the whole row in this entry
    dec.set_tensor(-1, rt.T_EMBEDDING, table)
    values, scales = dec.get_tensor(0, rt.T_WV)
    values[columns] = rng.integers(-1, 2, (2, cfg.dim))
    values[columns, 0] = 127
    scales[columns] = 5e35
    dec.set_tensor(0, rt.T_WV, values, scales)
    values, scales = dec.get_tensor(0, rt.T_WO)
    dec.set_tensor(0, rt.T_WO, values, np.full_like(scales, 1e-37))
    prompt = rng.integers(2, cfg.vocab_size, whole + 6)

    def last(n, at):
        p = prompt[:n].copy()
        if at is not None:
            p[at] = mark
        dec.prefill(p)
        return dec.last_hidden()

    for n, before in ((whole + 6, (5, 1)), (whole, (127, 84, 1))):
        want = last(n, None)
        assert np.all(np.isfinite(want))
        for back in before:
            np.testing.assert_array_equal(last(n, n - window - back), want, err_msg=str((n, back)))
        assert not np.array_equal(last(n, n - window), want)
    dec.close()


WIDE_FEED_FORWARD = """
import json, sys
import numpy as np
from kmll_b200 import runtime as rt
out = {}
for fmt in (rt.FORMAT_RS_I8, rt.FORMAT_W4G128):
    dec = rt.Decoder(rt.DecoderConfig(n_layers=2, dim=128, n_heads=2, n_kv_heads=1, head_dim=64, hidden_dim=16512, vocab_size=640, norm_eps=1e-6, max_seq_len=96, format=fmt))
    dec.init_random(3, 0.05)
    for n in (7, 33, 70):
        dec.prefill(np.arange(n) * 7 % 640)
        out[f"{fmt} {n}"] = dec.last_hidden().tolist()
    batch = rt.BatchDecoder(dec, 6)
    for slot in range(6):
        dec.prefill(np.arange(9) + slot)
        batch.adopt(slot)
    tokens, logits = batch.generate_greedy(3)
    out[f"{fmt} batch"] = logits.tolist()
    batch.close()
    dec.close()
print("RESULT " + json.dumps(out))
"""


def test_feed_forward_wider_than_a_block_holds(cuda):
    """A down projection of 16512 columns: more than the kernels that form SiLU(gate) * up in front of it keep in registers, so they
    read part of a row twice.  Prompts on either side of 32 rows against the oracle, and everything against the same
    without the tensor-core linears (KMLL_GEMM=0: gate, up, SiLU * up and the projection one after another)."""
    import json
    import os
    import subprocess
    import sys

    runs = []
    for env in ({}, {"KMLL_GEMM": "0"}):
        r = subprocess.run([sys.executable, "-c", WIDE_FEED_FORWARD], env=dict(os.environ, **env), capture_output=True, text=True, timeout=300,
                           cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
        assert r.returncode == 0, r.stderr[-2000:]
        runs.append(json.loads(next(line for line in r.stdout.splitlines() if line.startswith("RESULT "))[7:]))
    for key, want in runs[1].items():
        want, got = np.asarray(want), np.asarray(runs[0][key])
        assert np.max(np.abs(got - want)) <= 2e-4 * max(float(np.max(np.abs(want))), 1.0), key
    for fmt in (rt.FORMAT_RS_I8, rt.FORMAT_W4G128):
        cfg = rt.DecoderConfig(n_layers=2, dim=128, n_heads=2, n_kv_heads=1, head_dim=64, hidden_dim=16512, vocab_size=640, norm_eps=1e-6, max_seq_len=96, format=fmt)
        dec = make(cfg, seed=3)
        for n in (7, 33):
            ora = OracleDecoder(cfg, dec)
            ora.prefill(np.arange(n) * 7 % 640)
            assert np.max(np.abs(np.asarray(runs[0][f"{fmt} {n}"]) - ora.hidden)) <= 2e-4 * max(float(np.max(np.abs(ora.hidden))), 1.0), (fmt, n)
        dec.close()


@pytest.mark.parametrize("window", [1, 20, 70])
def test_f32_prompt_attention_window_keeps_non_finite_values_out(cuda, window):
    """fused = 0, one layer: the last row's hidden state does not change when a token before its window turns into NaN (the
    tile of keys that holds the window's start holds that token too), and does when the window reaches it."""
    cfg = tiny(rt.FORMAT_RS_I8, False, n_layers=1, max_seq_len=160, sliding_window=window)
    dec = make(cfg)
    table = dec.get_tensor(-1, rt.T_EMBEDDING).copy()
    table[639] = 0x7FC0
    dec.set_tensor(-1, rt.T_EMBEDDING, table)
    prompt = np.random.default_rng(window).integers(0, 639, 139)
    dec.prefill(prompt)
    want = dec.last_hidden()
    assert np.isfinite(want).all()
    poisoned = prompt.copy()
    poisoned[138 - window] = 639
    dec.prefill(poisoned)
    assert np.array_equal(dec.last_hidden(), want)
    poisoned[139 - window] = 639
    dec.prefill(poisoned)
    assert not np.isfinite(dec.last_hidden()).any()
    dec.close()


@pytest.mark.parametrize("kv_bf16", [False, True])
def test_long_context_fused_step_matches_oracle(cuda, kv_bf16):
    """A cache of 1300 positions x 8 KV heads: the fused batch-1 step plans slices of 128 positions (8 stages of 16, one
    per warp) and attends through the tensor-core kernel for the f32 cache as well (operands split into two bf16 parts,
    about 2^-17 per product): the f32 tolerances of the other tests hold."""
    cfg = tiny(rt.FORMAT_W4G128, True, n_heads=8, n_kv_heads=8, head_dim=64, dim=512, max_seq_len=1300, kv_bf16=kv_bf16)
    dec = make(cfg)
    prompt = np.random.default_rng(21).integers(0, cfg.vocab_size, 1210)
    check_against_oracle(dec, cfg, prompt, 6, batched_prefill=True, **(BF16_KV_BOUND if kv_bf16 else {}))
    dec.close()


@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("batched_prefill", [False, True])
def test_single_token_prompt(cuda, kv_bf16, batched_prefill):
    """The shortest sequences: a one-token prompt (one query row, one key), then steps whose blocks hold only the row
    being written plus a handful of cached rows."""
    cfg = tiny(rt.FORMAT_RS_I8, True, n_heads=8, n_kv_heads=2, head_dim=128, dim=256, max_seq_len=40, kv_bf16=kv_bf16)
    dec = make(cfg)
    check_against_oracle(dec, cfg, np.asarray([7]), 6, batched_prefill=batched_prefill, **(BF16_KV_BOUND if kv_bf16 else {}))
    dec.close()


BF16_KV_BOUND = dict(hid_tol=2e-3, min_margin=1e-2, logit_tol=5e-3)


@pytest.mark.parametrize("fmt", [rt.FORMAT_RS_I8, rt.FORMAT_W4G128])
@pytest.mark.parametrize("head_dim,n_heads,n_kv", [(64, 4, 2), (128, 8, 1), (128, 8, 2)])
@pytest.mark.parametrize("batched_prefill", [False, True])
def test_bf16_kv_cache_matches_oracle(cuda, fmt, head_dim, n_heads, n_kv, batched_prefill):
    """kv_bf16: the oracle rounds the K / V rows it stores to bf16 (nearest-even) and is otherwise unchanged.  The bound
    is the option's own: a K / V value that the two sides compute a few f32 ulps apart can fall on either side of a bf16
    rounding tie, which moves that cache element by one bf16 ulp (2^-8 relative) - hidden state within 2e-3 of its scale,
    logits within 5e-3, tokens compared while the oracle's top-2 margin is at least 1e-2.  The sequence crosses a
    64-position tile so that staged rows, the row being written and both prefill paths are covered.  The cache bytes are
    half those of the f32 cache."""
    cfg = tiny(fmt, True, n_heads=n_heads, n_kv_heads=n_kv, head_dim=head_dim, dim=256, max_seq_len=160, kv_bf16=True)
    dec = make(cfg)
    ref = make(tiny(fmt, True, n_heads=n_heads, n_kv_heads=n_kv, head_dim=head_dim, dim=256, max_seq_len=160))
    assert dec.kv_bytes * 2 == ref.kv_bytes
    ref.close()
    rng = np.random.default_rng(11)
    prompt = rng.integers(0, cfg.vocab_size, 61)
    check_against_oracle(dec, cfg, prompt, 8, batched_prefill=batched_prefill, **BF16_KV_BOUND)
    dec.close()


@pytest.mark.parametrize("fused,rotary_dim", [(False, None), (True, 32), (False, 32)])
def test_bf16_kv_cache_on_the_other_step_forms(cuda, fused, rotary_dim):
    """The operator-by-operator step and the partial-rotary step (RoPE + cache write in a kernel of their own) over a
    bf16 cache."""
    cfg = tiny(rt.FORMAT_W4G128, fused, rotary_dim=rotary_dim, max_seq_len=96, kv_bf16=True)
    dec = make(cfg)
    prompt = np.random.default_rng(5).integers(0, cfg.vocab_size, 66)
    check_against_oracle(dec, cfg, prompt, 5, batched_prefill=fused, **BF16_KV_BOUND)
    dec.close()


@pytest.mark.parametrize("fmt", [rt.FORMAT_RS_I8, rt.FORMAT_W4G128])
def test_batched_prefill_matches_oracle_and_token_loop(cuda, fmt):
    cfg = tiny(fmt, True, n_heads=8, n_kv_heads=2, head_dim=128, dim=256, max_seq_len=64)
    dec = make(cfg)
    rng = np.random.default_rng(3)
    prompt = rng.integers(0, cfg.vocab_size, 21)
    check_against_oracle(dec, cfg, prompt, 5, batched_prefill=True)
    # batched prefill and the per-token path leave the same pending token and (nearly) the same hidden state
    dec.prefill(prompt)
    a_top, a_hid = dec.next_top(), dec.last_hidden()
    dec.prefill(prompt, token_loop=True)
    b_top, b_hid = dec.next_top(), dec.last_hidden()
    assert rt.unpack_top1(a_top)[0] == rt.unpack_top1(b_top)[0]
    assert np.max(np.abs(a_hid - b_hid)) <= 2e-4 * max(np.max(np.abs(b_hid)), 1.0)
    dec.close()


def test_prompt_scratch_is_no_decoders_and_is_given_back(cuda):
    """Growing and shorter prompts in shared scratch give what they give in a fresh decoder; byte counts stay, one buffer serves two
    decoders, and nothing is held once it is released."""
    cfg = tiny(rt.FORMAT_W4G128, hidden_dim=8192, max_seq_len=600)
    rng = np.random.default_rng(8)
    prompts = [rng.integers(0, cfg.vocab_size, n) for n in (40, 600, 7, 300, 1)]
    want = []
    for p in prompts:
        dec = make(cfg)
        rt.release_scratch()
        dec.prefill(p)
        want.append(dec.last_hidden())
        dec.close()
    rt.release_scratch()
    decs = [make(cfg), make(cfg)]
    resident = decs[0].resident_bytes
    free = torch.cuda.mem_get_info()[0]
    for dec in decs:
        for p, w in zip(prompts, want):
            dec.prefill(p)
            assert np.array_equal(dec.last_hidden(), w)
        assert dec.resident_bytes == resident
    held = free - torch.cuda.mem_get_info()[0]
    rows = 600 * 4 * (2 * 256 + 3 * 256 + 2 * 128 + 2 * 8192)  # of the longest prompt
    assert rows <= held <= 1.5 * rows + (32 << 20)  # planes and partial tiles of the linears beside them; once, not twice
    assert rt.release_scratch() >= rows and rt.release_scratch() == 0
    assert torch.cuda.mem_get_info()[0] == free
    decs[0].prefill(prompts[1])
    assert np.array_equal(decs[0].last_hidden(), want[1])
    for dec in decs:
        dec.close()


def test_prompt_scratch_above_its_bound_is_not_kept(cuda):
    cfg = tiny(rt.FORMAT_RS_I8, n_layers=1, dim=64, n_heads=1, n_kv_heads=1, hidden_dim=16384, max_seq_len=14000)
    dec = make(cfg)
    prompt = np.random.default_rng(4).integers(0, cfg.vocab_size, 14000)  # 14000 x (2 x 16384 x 4 + 16384 x 4) bytes and more
    dec.prefill(prompt)
    rt.release_scratch()
    free = torch.cuda.mem_get_info()[0]
    dec.prefill(prompt)
    assert torch.cuda.mem_get_info()[0] == free and rt.release_scratch() == 0
    assert np.isfinite(dec.last_hidden()).all()
    dec.close()


def test_kept_prompt_scratch_makes_room_for_a_batch(cuda):
    """A batch that fits the GPU only without the kept scratch can be created."""
    cfg = tiny(rt.FORMAT_RS_I8, n_layers=1, dim=64, n_heads=1, n_kv_heads=1, hidden_dim=16384, max_seq_len=8000)
    dec = make(cfg)
    dec.prefill(np.arange(8000) % cfg.vocab_size)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    kept = rt.release_scratch()
    assert kept > 1 << 30
    dec.prefill(np.arange(8000) % cfg.vocab_size)
    hold = torch.empty(free - (kept >> 2), dtype=torch.uint8, device="cuda")
    other = rt.DecoderConfig(**{**cfg.__dict__, "max_seq_len": kept // 2 // (2 * 64 * 4)})  # its caches: half of the kept scratch
    try:
        second = make(other)
        assert rt.release_scratch() == 0
        second.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    dec.close()


def test_prompts_of_two_threads_have_scratch_of_their_own(cuda):
    from concurrent.futures import ThreadPoolExecutor

    cfg = tiny(rt.FORMAT_W4G128, hidden_dim=2048, max_seq_len=300)
    rng = np.random.default_rng(12)
    prompts = [rng.integers(0, cfg.vocab_size, n) for n in (300, 45, 120, 9) * 6]

    def all_of(dec, order):
        with torch.cuda.stream(torch.cuda.Stream()):
            got = {}
            for i in order:
                dec.prefill(prompts[i])
                got[i] = dec.last_hidden()
            return got

    decs = [make(cfg) for _ in range(3)]
    want = all_of(decs[0], range(len(prompts)))
    with ThreadPoolExecutor(3) as pool:
        for got in pool.map(all_of, decs, [range(24), range(23, -1, -1), range(24)]):
            assert all(np.array_equal(got[i], want[i]) for i in range(24))
    for dec in decs:
        dec.close()


def test_fused_and_unfused_paths_agree(cuda):
    prompt = np.arange(1, 8)
    outs = []
    for fused in (True, False):
        cfg = tiny(rt.FORMAT_W4G128, fused)
        dec = make(cfg, seed=5)
        dec.prefill(prompt, token_loop=True)
        outs.append(dec.generate_greedy(10))
        dec.close()
    assert np.array_equal(outs[0][0], outs[1][0])
    assert np.max(np.abs(outs[0][1] - outs[1][1])) <= 1e-3


def test_step_host_equals_graph_loop_and_is_repeatable(cuda):
    cfg = tiny(rt.FORMAT_W4G128)
    dec = make(cfg, seed=7)
    prompt = np.array([5, 17, 300, 2])
    dec.prefill(prompt)
    tokens, logits = dec.generate_greedy(8)
    dec.prefill(prompt)
    packed = dec.next_top()
    via_host = []
    for _ in range(8):
        tok, logit = rt.unpack_top1(packed)
        via_host.append((tok, logit))
        packed = dec.step_host(tok)
    assert [t for t, _ in via_host] == tokens.tolist()
    assert np.array_equal(np.array([l for _, l in via_host], dtype=F), logits)
    # the decode loop is deterministic: a second run gives bit-identical logits
    dec.prefill(prompt)
    tokens2, logits2 = dec.generate_greedy(8)
    assert np.array_equal(tokens, tokens2) and np.array_equal(logits, logits2)
    dec.close()


def test_tied_embeddings_use_the_embedding_table_as_output(cuda):
    import oracle
    for fmt in (rt.FORMAT_RS_I8, rt.FORMAT_W4G128):
        cfg = tiny(fmt)
        dec = make(cfg, tie=True)
        emb = dec.get_tensor(-1, rt.T_EMBEDDING)
        values, scales = dec.get_tensor(-1, rt.T_OUTPUT)
        if fmt == rt.FORMAT_RS_I8:
            q, sc = oracle.rs_i8_quantize(emb)
            assert np.array_equal(values, q) and np.array_equal(scales, sc)
        else:
            p, gs = oracle.w4_quantize(oracle.bf16_to_f32(emb))
            assert np.array_equal(values, p) and np.array_equal(scales, gs)
        dec.close()


def test_runtime_errors(cuda):
    cfg = tiny(rt.FORMAT_W4G128, max_seq_len=8)
    dec = make(cfg)
    with pytest.raises(KmllError):
        dec.generate_greedy(1)  # runtime must be prefilled before generation
    with pytest.raises(KmllError):
        dec.prefill(np.arange(9))  # longer than max_seq_len
    with pytest.raises(KmllError):
        dec.prefill(np.array([cfg.vocab_size]))  # token out of range
    dec.prefill(np.arange(5))
    with pytest.raises(KmllError):
        dec.generate_greedy(4)  # position would exceed max sequence length
    dec.generate_greedy(3)
    dec.close()
    with pytest.raises(KmllError):
        rt.Decoder(tiny(rt.FORMAT_W4G128, n_heads=3))  # heads not divisible
    with pytest.raises(KmllError):
        rt.Decoder(tiny(rt.FORMAT_W4G128, dim=200))  # not a multiple of the group size


def test_qwen2_shape_slice(cuda):
    """Qwen2-0.5B geometry (hidden 896, 14/2 heads of 64, intermediate 4864, tied embeddings) with 2 layers and a
    small vocabulary: exercises K = 896 and 4864 (not multiples of the 2 KB stage) against the oracle."""
    cfg = rt.DecoderConfig(n_layers=2, dim=896, n_heads=14, n_kv_heads=2, head_dim=64, hidden_dim=4864, vocab_size=1024,
                           rope_theta=1e6, norm_eps=1e-6, max_seq_len=40, format=rt.FORMAT_W4G128)
    dec = make(cfg, seed=2, std=0.02, tie=True)
    rng = np.random.default_rng(2)
    check_against_oracle(dec, cfg, rng.integers(0, cfg.vocab_size, 12), 4, batched_prefill=True)
    dec.close()


def test_timeline_attach_and_detach_recapture_the_step_graph(cuda):
    """The per-token CUDA graph bakes the timeline slots of its launches: after the buffer is detached the decoder must
    capture the graph again, so replays leave the (possibly freed) buffer alone; attaching later must trace again."""
    import ctypes as C
    from kmll_b200 import lib as klib
    L = klib.load()
    cfg = tiny(rt.FORMAT_W4G128)
    dec = make(cfg, seed=7)
    prompt = np.array([5, 17, 300, 2])
    dec.prefill(prompt)
    ref_tokens, _ = dec.generate_greedy(6)  # graph captured with no buffer attached
    buf = torch.zeros(1 << 16, dtype=torch.int64, device="cuda")
    count = C.c_int(0)
    klib.check(L.kmll_trace_attach(C.c_void_p(buf.data_ptr()), buf.numel() * 8))
    dec.prefill(prompt)
    tokens, _ = dec.generate_greedy(6)
    torch.cuda.synchronize()
    klib.check(L.kmll_trace_launches(None, None, None, 0, C.byref(count)))
    assert count.value > 0 and int(torch.count_nonzero(buf)) > 0, "attaching after the first capture must trace the step"
    assert tokens.tolist() == ref_tokens.tolist()
    klib.check(L.kmll_trace_attach(None, 0))
    buf.zero_()
    dec.prefill(prompt)
    tokens, _ = dec.generate_greedy(6)
    torch.cuda.synchronize()
    assert int(torch.count_nonzero(buf)) == 0, "a detached buffer must not be written by later replays"
    assert tokens.tolist() == ref_tokens.tolist()
    dec.close()


@pytest.mark.parametrize("fmt", [rt.FORMAT_RS_I8, rt.FORMAT_W4G128])
def test_archive_round_trip_gives_the_same_model(cuda, fmt, tmp_path):
    """Export a decoder's linear tensors in kmll's archive layout, load them into a fresh decoder (norms and embeddings
    travel separately, as in kmll where they stay in the checkpoint): the tensors are bit-identical and the greedy
    tokens equal the in-memory model's."""
    cfg = tiny(fmt)
    dec = make(cfg, seed=11)
    prompt = np.array([7, 300, 12, 5, 99])
    dec.prefill(prompt)
    ref_tokens, ref_logits = dec.generate_greedy(8)
    d = str(tmp_path / "export")
    dec.export_archive(d, "/models/demo.safetensors")
    fresh = rt.Decoder(cfg)
    for layer in range(cfg.n_layers):
        fresh.set_tensor(layer, rt.T_ATTENTION_NORM, dec.get_tensor(layer, rt.T_ATTENTION_NORM))
        fresh.set_tensor(layer, rt.T_FFN_NORM, dec.get_tensor(layer, rt.T_FFN_NORM))
    fresh.set_tensor(-1, rt.T_FINAL_NORM, dec.get_tensor(-1, rt.T_FINAL_NORM))
    fresh.set_tensor(-1, rt.T_EMBEDDING, dec.get_tensor(-1, rt.T_EMBEDDING))
    fresh.load_archive(d, "/models/demo.safetensors")
    for layer, tensor in ((0, rt.T_WQ), (1, rt.T_W2), (-1, rt.T_OUTPUT)):
        a, b = dec.get_tensor(layer, tensor), fresh.get_tensor(layer, tensor)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1].view(np.uint8), b[1].view(np.uint8))
    fresh.prefill(prompt)
    tokens, logits = fresh.generate_greedy(8)
    assert np.array_equal(tokens, ref_tokens) and np.array_equal(logits, ref_logits)
    with pytest.raises(KmllError):
        fresh.load_archive(d, "/models/another.safetensors")
    dec.close()
    fresh.close()
