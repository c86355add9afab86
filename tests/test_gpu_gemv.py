"""tomos_gemv (every storage type, tier, layout, transpose, beta) against
an FP64 product of the values the tier reads (oracle decode), and against
the reference's own CPU FP32_16 tiers."""
import ctypes
import os

import numpy as np
import pytest
import torch

import tomos_b200 as tb
from tomos_b200 import _capi as C
from gpu_util import to_dense, decoded, cuda

GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
pytestmark = pytest.mark.gpu

L = tb.Layout
NT = tb.NumericType
CASES = [(NT.FP32, tb.Tier.AUTO, False), (NT.FP32_16, tb.Tier.HALF, False),
         (NT.FP32_16, tb.Tier.ACCURATE, False), (NT.FP32_BF16, tb.Tier.HALF, False),
         (NT.FP32_BF16, tb.Tier.ACCURATE, False), (NT.FP32_BF16, tb.Tier.ACCURATE, True)]


def run(A, trans, tier, x, alpha, beta, y0):
    y = cuda(y0)
    tb.mv_apply(tb.Device.CUDA, trans, alpha, A, cuda(x), beta, y, tier=tier)
    return y.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("numeric,tier,rounded", CASES)
@pytest.mark.parametrize("layout", [L.ROW_MAJOR, L.COL_MAJOR])
@pytest.mark.parametrize("shape", [(1, 1), (7, 5), (33, 257), (1000, 37), (4097, 300)])
def test_gemv_vs_fp64(orc, numeric, tier, rounded, layout, shape):
    rng = np.random.default_rng(hash((shape, int(layout))) % 2 ** 32)
    m, n = shape
    A0 = (rng.standard_normal((m, n)) * np.where(rng.random((m, n)) < 0.05, 1e-6, 1.0)).astype(np.float32)
    A = to_dense(A0, layout, numeric, pad=2, rounded=rounded)
    Ad = decoded(orc, A, tier)
    acc64 = tier == tb.Tier.ACCURATE
    for trans in (tb.NO_TRANSPOSE, tb.TRANSPOSE):
        M = Ad if trans == tb.NO_TRANSPOSE else Ad.T
        x = rng.standard_normal(M.shape[1]).astype(np.float32)
        for beta in (0.0, 0.5):
            y0 = rng.standard_normal(M.shape[0]).astype(np.float32)
            if beta == 0.0:
                y0[:] = np.nan  # beta == 0 must not read y
            ref = 1.5 * (M @ x.astype(np.float64)) + (beta * y0.astype(np.float64) if beta else 0.0)
            scale = 1.5 * (np.abs(M) @ np.abs(x.astype(np.float64))) + abs(beta) * np.abs(np.nan_to_num(y0))
            got = run(A, trans, tier, x, 1.5, beta, y0)
            tol = (2e-6 if acc64 else 2e-5) * scale + 1e-30
            assert np.all(np.abs(got - ref) <= tol + 1e-7 * np.abs(ref)), (trans, beta)


@pytest.mark.parametrize("numeric,tier,rounded", CASES + [(NT.FP16, tb.Tier.AUTO, False)])
@pytest.mark.parametrize("m,n,pad", [(5001, 9, 0), (3, 64, 0), (4999, 256, 0), (17, 258, 0), (2049, 65, 0),
                                     (1501, 777, 0), (700, 1025, 0), (40003, 7, 1), (8200, 600, 4),
                                     (33000, 100, 0), (2000, 127, 0), (2000, 128, 0), (24001, 65, 0),
                                     (10001, 64, 0), (40011, 513, 0), (23, 999, 0), (25, 999, 0)])
@pytest.mark.parametrize("layout", [L.ROW_MAJOR, L.COL_MAJOR])
def test_gemv_line_shapes(orc, numeric, tier, rounded, m, n, pad, layout):
    """Narrow and unaligned lines (the direct pass), few long lines (a CTA a
    segment, chunks of eight lines), aligned or not, both ways."""
    rng = np.random.default_rng(m + n)
    A0 = (rng.standard_normal((m, n)) * np.where(rng.random((m, n)) < 0.05, 1e-6, 1.0)).astype(np.float32)
    if numeric == NT.FP16:
        A = tb.pack(to_dense(A0, layout, pad=pad), NT.FP16)
        Ad = A.view().double().cpu().numpy()
    else:
        A = to_dense(A0, layout, numeric, pad=pad, rounded=rounded)
        Ad = decoded(orc, A, tier)
    for trans in (tb.NO_TRANSPOSE, tb.TRANSPOSE):
        M = Ad if trans == tb.NO_TRANSPOSE else Ad.T
        x = rng.standard_normal(M.shape[1]).astype(np.float32)
        for beta in (0.0, -0.5):
            y0 = rng.standard_normal(M.shape[0]).astype(np.float32) if beta else np.full(M.shape[0], np.nan, np.float32)
            ref = 1.5 * (M @ x.astype(np.float64)) + (beta * y0.astype(np.float64) if beta else 0.0)
            scale = 1.5 * (np.abs(M) @ np.abs(x.astype(np.float64))) + abs(beta) * np.abs(np.nan_to_num(y0))
            got = run(A, trans, tier, x, 1.5, beta, y0)
            # exact tiers: FP32 runs of at most 8 at worst, then one rounding
            tol = (2e-6 if tier == tb.Tier.ACCURATE else 2e-5) * scale + 1e-30
            assert np.all(np.abs(got - ref) <= tol + 1e-7 * np.abs(ref)), (trans, beta)


@pytest.mark.parametrize("offset", [0, 4])
def test_few_long_dots_scratch_alignment(offset):
    """Dots of few, long lines with a scratch on 8 bytes (FP64 partials of a
    line's segments) and on 4 bytes only (a warp a line)."""
    rng = np.random.default_rng(5)
    m, n = 40000, 3
    A0 = rng.standard_normal((m, n)).astype(np.float32)
    A, x = to_dense(A0, L.COL_MAJOR), rng.standard_normal(m).astype(np.float32)
    lib, d = C.lib(), A.desc()
    nb = lib.tomos_gemv_scratch_bytes(ctypes.byref(d), int(tb.TRANSPOSE))
    assert nb > 0
    scratch = torch.empty(nb + 8, dtype=torch.uint8, device="cuda")
    xt, y = torch.from_numpy(x).cuda(), torch.empty(n, device="cuda")
    C.check(lib.tomos_gemv(int(tb.TRANSPOSE), 1.0, ctypes.byref(d), int(tb.Tier.AUTO), xt.data_ptr(), 0.0,
                           y.data_ptr(), scratch.data_ptr() + offset, nb, None), "gemv")
    torch.cuda.synchronize()
    ref = A0.astype(np.float64).T @ x
    # FP32 products and sums of at most m / 32 terms a lane
    tol = (m / 32 + 40) * 6e-8 * (np.abs(A0).astype(np.float64).T @ np.abs(x))
    assert np.all(np.abs(y.cpu().numpy() - ref) <= tol)


def test_fp32_16_tiers_vs_reference_cpu(orc):
    """The reference's CPU tiers (fp32_16_kernels.cpp): our HALF tier is its
    'fast' tier (fp32_16_half_only decode, wide accumulation), ACCURATE its
    exact tier.  Reference tolerances (test_fp32_16.cpp:178-182) plus a
    tight FP32-rounding bound."""
    g = np.load(os.path.join(GOLD, "mv_fp32_16.npz"))
    A = to_dense(g["A"], L.COL_MAJOR, NT.FP32_16)
    for trans, x, key in ((tb.NO_TRANSPOSE, g["x"], "y"), (tb.TRANSPOSE, g["xt"], "yt")):
        half = run(A, trans, tb.Tier.HALF, x, 1.0, 0.0, np.zeros(len(g[key + "1"]), np.float32))
        acc = run(A, trans, tb.Tier.ACCURATE, x, 1.0, 0.0, np.zeros(len(g[key + "2"]), np.float32))
        fast_ref, acc_ref = g[key + "1"].astype(np.float64), g[key + "2"].astype(np.float64)
        assert np.all(np.abs(half - fast_ref) <= 0.05 * np.abs(fast_ref) + 0.05)
        assert np.all(np.abs(acc - acc_ref) <= 1e-3 * np.abs(acc_ref) + 1e-4)
        np.testing.assert_allclose(half, fast_ref, rtol=1e-5, atol=1e-4)
        np.testing.assert_allclose(acc, acc_ref, rtol=1e-6, atol=1e-5)


def test_unregistered_compute_type_raises():
    A = to_dense(np.ones((4, 4), np.float32), L.COL_MAJOR)
    y = cuda(np.zeros(4, np.float32))
    with pytest.raises(tb.TomosError):
        tb.mv_apply(tb.Device.CUDA, tb.NO_TRANSPOSE, 1.0, A, cuda(np.ones(4)), 0.0, y,
                    compute_type=NT.FP16)
