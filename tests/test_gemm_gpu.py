"""Batched quantized linear on the tensor cores (tcgen05, caller-owned workspace) against the CPU oracle: the shapes of
the quantized GEMM sweep (M = 64, 256; (N, K) = (3584, 3584), (18944, 3584), (3584, 18944), a slice of (152064, 3584)),
prefill shapes of the Mistral-7B architecture, ragged sizes, both weight formats.  Same bounds as every other linear:
kmll's max_abs <= 1e-4 sqrt(K) (src/main.rs:4306) and 1e-4 relative to the largest output."""
import numpy as np
import pytest
import torch

import oracle
from kmll_b200 import ops
from test_ops_gpu import F, assert_close, dev, host, i8_weight, w4_weight

pytestmark = pytest.mark.gpu

SHAPES = [(5, 300, 512), (16, 4096, 4096), (33, 700, 4096), (64, 3584, 3584), (256, 3584, 3584), (64, 18944, 3584),
          (256, 3584, 18944), (64, 4736, 3584), (300, 1000, 256), (2048, 1024, 4096), (128, 4096, 14336)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_gemm_w4_vs_oracle(cuda, m, n, k):
    rng = np.random.default_rng(m + n + k)
    _, packed, gs, w = w4_weight(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(F)
    x[0, :] *= F(1e-3)  # rows of very different magnitude: the scale is per row
    x[m - 1, :] *= F(1e3)
    ref = oracle.w4_linear_batched(x, packed, gs)
    ws = ops.linear_batched_workspace(m, k)
    assert ws is not None
    got = host(ops.linear_batched(dev(x), w, m, k, n, workspace=ws))
    assert_close(got[m // 2], ref[m // 2], k, f"w4 gemm {m}x{n}x{k} row {m // 2}")  # an unscaled row: kmll's absolute bound
    scale = np.maximum(np.max(np.abs(ref), axis=1, keepdims=True), 1e-30)
    assert float(np.max(np.abs(got - ref) / scale)) <= 1e-4  # every row, relative to its own largest output


# 5 to 32 rows of x: the persistent small-batch kernel (byte digits, s8 x s8 MMAs, group scale after the MMA); shapes
# with a ragged last row tile, one row tile only, split K (few row tiles) and no split (many), 16 and 32 row blocks
SMALL = [(5, 100, 128), (16, 1024, 4096), (17, 4097, 1024), (32, 14336, 4096), (16, 4096, 14336), (8, 18944, 3584), (24, 3584, 18944),
         (16, 32000, 4096)]


@pytest.mark.parametrize("m,n,k", SMALL)
def test_small_batch_w4_vs_oracle(cuda, m, n, k):
    rng = np.random.default_rng(m * 3 + n + k)
    _, packed, gs, w = w4_weight(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(F)
    x[0, :] *= F(1e-3)
    x[m - 1, :] *= F(1e3)
    x[1, 7] = F(300.0)  # an activation far above the rest of its row
    ref = oracle.w4_linear_batched(x, packed, gs)
    ws = ops.linear_batched_workspace(m, k)
    r = rng.normal(0, 1, (m, n)).astype(F)
    got = host(ops.linear_batched(dev(x), w, m, k, n, workspace=ws))
    assert_close(got[m // 2], ref[m // 2], k, f"small batch {m}x{n}x{k} row {m // 2}")
    scale = np.maximum(np.max(np.abs(ref), axis=1, keepdims=True), 1e-30)
    assert float(np.max(np.abs(got - ref) / scale)) <= 1e-4
    again = host(ops.linear_batched(dev(x), w, m, k, n, workspace=ws))
    assert np.array_equal(got, again)  # split-K partials are added in split order: bit-identical from call to call
    del r


@pytest.mark.parametrize("m,n,k", [(5, 100, 256), (16, 1024, 4096), (17, 4097, 1024), (32, 14336, 4096), (16, 4096, 14336), (9, 700, 320),
                                   (16, 32000, 4096)])
def test_small_batch_i8_vs_oracle(cuda, m, n, k):
    """RS-I8, 5 to 32 rows of x: the int8 rows are MMA operands as they lie (K = 320: a partial last group)."""
    rng = np.random.default_rng(m * 5 + n + k)
    _, q, sc, w = i8_weight(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(F)
    x[0, :] *= F(1e-3)
    x[m - 1, :] *= F(1e3)
    x[1, 7] = F(300.0)
    ref = oracle.rs_i8_linear_batched(x, q, sc)
    ws = ops.linear_batched_workspace(m, k)
    got = host(ops.linear_batched(dev(x), w, m, k, n, workspace=ws))
    assert_close(got[m // 2], ref[m // 2], k, f"small batch i8 {m}x{n}x{k} row {m // 2}")
    scale = np.maximum(np.max(np.abs(ref), axis=1, keepdims=True), 1e-30)
    assert float(np.max(np.abs(got - ref) / scale)) <= 1e-4
    assert np.array_equal(got, host(ops.linear_batched(dev(x), w, m, k, n, workspace=ws)))


@pytest.mark.parametrize("m,n,k", SHAPES[:5] + [(64, 1000, 896), (2048, 1024, 4096)])
def test_gemm_i8_vs_oracle(cuda, m, n, k):
    rng = np.random.default_rng(m + n + k + 1)
    _, q, sc, w = i8_weight(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(F)
    ref = oracle.rs_i8_linear_batched(x, q, sc)
    got = host(ops.linear_batched(dev(x), w, m, k, n))
    scale = np.maximum(np.max(np.abs(ref), axis=1, keepdims=True), 1e-30)
    assert float(np.max(np.abs(got - ref) / scale)) <= 1e-4
    assert float(np.max(np.abs(got - ref))) <= 1e-4 * np.sqrt(k)


def test_gemm_qkv_and_is_deterministic(cuda):
    rng = np.random.default_rng(9)
    m, k = 96, 4096
    mats = [w4_weight(rng, rows, k) for rows in (4096, 1024, 1024)]
    x = rng.normal(0, 1, (m, k)).astype(F)
    xd = dev(x)
    q, kk, v = ops.linear_qkv_batched(xd, mats[0][3], mats[1][3], mats[2][3], m, k)
    for got, (_, packed, gs, _) in zip((q, kk, v), mats):
        ref = oracle.w4_linear_batched(x, packed, gs)
        assert float(np.max(np.abs(host(got) - ref))) <= 1e-4 * np.sqrt(k)
    q2, _, _ = ops.linear_qkv_batched(xd, mats[0][3], mats[1][3], mats[2][3], m, k)
    assert torch.equal(q, q2)


def test_small_batch_qkv_one_launch(cuda):
    """Three matrices of different heights share the digits of x and one persistent launch; RMSNorm fused in front."""
    rng = np.random.default_rng(11)
    m, k = 16, 4096
    mats = [w4_weight(rng, rows, k) for rows in (4096, 1000, 1000)]
    x = rng.normal(0, 1, (m, k)).astype(F)
    xd = dev(x)
    q, kk, v = ops.linear_qkv_batched(xd, mats[0][3], mats[1][3], mats[2][3], m, k)
    for got, (_, packed, gs, _) in zip((q, kk, v), mats):
        ref = oracle.w4_linear_batched(x, packed, gs)
        assert float(np.max(np.abs(host(got) - ref))) <= 1e-4 * np.sqrt(k)


def test_gemm_without_workspace_still_works(cuda):
    """No workspace: the call falls back to passes of the streaming kernel (4 rows of x each) and gives the same result."""
    rng = np.random.default_rng(10)
    m, n, k = 9, 256, 512
    _, packed, gs, w = w4_weight(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(F)
    ref = oracle.w4_linear_batched(x, packed, gs)
    from kmll_b200.lib import check, load
    out = torch.empty((m, n), device="cuda")
    xd = dev(x)
    check(load().kmll_linear_batched_w4g128(torch.cuda.current_stream().cuda_stream, xd.data_ptr(), w.packed.data_ptr(), w.gscales.data_ptr(), m, k,
                                            n, None, out.data_ptr()))
    assert float(np.max(np.abs(host(out) - ref))) <= 1e-4 * np.sqrt(k)


# K cut into pieces and not; a call's own counters are clear whatever the workspace held
@pytest.mark.parametrize("fmt", ["w4", "i8"])
@pytest.mark.parametrize("m,n,k", [(5, 130, 4096), (16, 3000, 2048), (32, 128, 16512), (8, 40000, 256), (48, 300, 8192)])
def test_workspace_contents_do_not_matter(cuda, fmt, m, n, k):
    rng = np.random.default_rng(m + n)
    w = (w4_weight if fmt == "w4" else i8_weight)(rng, n, k)[3]
    x = dev(rng.normal(0, 1, (m, k)).astype(F))
    ws = ops.linear_batched_workspace(m, k)
    want = None
    for fill in (0, 1, 0xff, 3):
        ws.fill_(fill)
        got = host(ops.linear_batched(x, w, m, k, n, workspace=ws))
        want = got if want is None else want
        assert np.array_equal(got, want)
        again = host(ops.linear_batched(x, w, m, k, n, workspace=ws))  # (and what a call leaves there)
        assert np.array_equal(again, want)
    w64, x64 = host(w.dequantize()).astype(np.float64).reshape(n, k), host(x).astype(np.float64)
    assert np.all(np.abs(want.reshape(m, n) - x64 @ w64.T) <= 1e-5 * (np.abs(x64) @ np.abs(w64).T))


# 33 and more rows of x: pairs of blocks, 256 weight rows against up to 256 rows of x.  One row of weights, one k-tile, one group,
# both sides of the one-MMA form (128 rows of x), ragged last tiles on either side, split K, several units per pair.
PAIR = [("w4", 33, 1, 128), ("w4", 128, 257, 256), ("w4", 129, 300, 384), ("w4", 256, 256, 384), ("w4", 257, 255, 128), ("w4", 40, 600, 16384),
        ("w4", 700, 3000, 1152), ("i8", 33, 1, 64), ("i8", 65, 300, 192), ("i8", 300, 257, 320), ("i8", 48, 130, 8192), ("i8", 1100, 5000, 128)]


@pytest.mark.parametrize("fmt,m,n,k", PAIR)
def test_pair_gemm_error_bound(cuda, fmt, m, n, k):
    """Against 64-bit sums of the dequantized weights.  Bound per output: two binary16 planes of x (2^-22 of every product) and
    f32 sums in steps of 16 columns (2^-23 of the partial sum each), times sum |w x|."""
    rng = np.random.default_rng(m * 7 + n + k)
    x = rng.normal(0, 1, (m, k)).astype(F)
    x[m // 3] *= F(1e-3)
    if fmt == "w4":
        w = w4_weight(rng, n, k)[3]
    else:
        w = i8_weight(rng, n, k)[3]
    w64 = host(w.dequantize()).astype(np.float64).reshape(n, k)
    x64 = x.astype(np.float64)
    got = host(ops.linear_batched(dev(x), w, m, k, n, workspace=ops.linear_batched_workspace(m, k))).reshape(m, n)
    bound = (2.0 ** -22 + (k / 16 + 16) * 2.0 ** -23) * (np.abs(x64) @ np.abs(w64).T) + 1e-30
    assert np.all(np.abs(got - x64 @ w64.T) <= bound)
    # That bound lets a lost plane of x pass at long K.  As a whole, rows of x of equal weight: half a bit of the planes (2^-22) and of each
    # step of the sums, W4 eight to a group and one per group, RS-I8 one per 16 columns, half of them in either accumulator.  Without the low plane: 1.4e-4.
    steps = 8 + k / 128 if fmt == "w4" else k / 32
    length = np.linalg.norm(x64, axis=1)[:, None]
    off = np.linalg.norm((got - x64 @ w64.T) / length) / np.linalg.norm(x64 @ w64.T / length)
    assert off <= 2.0 ** -22 + steps * 2.0 ** -23
    again = host(ops.linear_batched(dev(x), w, m, k, n, workspace=ops.linear_batched_workspace(m, k))).reshape(m, n)
    assert np.array_equal(got, again)


def test_pair_gemm_three_matrices(cuda):
    """Matrices of different, ragged heights in one launch, against 64-bit sums, bound as above."""
    rng = np.random.default_rng(12)
    m, k = 130, 512
    mats = [w4_weight(rng, rows, k)[3] for rows in (513, 300, 300)]
    xd = dev(rng.normal(0, 1, (m, k)).astype(F))
    for got, w in zip(ops.linear_qkv_batched(xd, *mats, m, k), mats):
        w64 = host(w.dequantize()).astype(np.float64).reshape(-1, k)
        x64 = host(xd).astype(np.float64)
        bound = (2.0 ** -22 + (k / 16 + 16) * 2.0 ** -23) * (np.abs(x64) @ np.abs(w64).T) + 1e-30
        assert np.all(np.abs(host(got).reshape(m, -1) - x64 @ w64.T) <= bound)
