"""Bit widening of finite FP32 / BF16 values in the streaming passes: exact for
every BF16 pattern and sampled FP32 ones (numpy restatement of the device
expression), and fits with non-finite predictors still fail."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W


def test_widening_is_exact():
    rng = np.random.default_rng(0)
    bits = np.concatenate([np.arange(65536, dtype=np.uint32) << 16,
                           rng.integers(0, 2 ** 32, 500_000, dtype=np.uint64).astype(np.uint32)])
    v = bits.view(np.float32)
    bits, v = bits[np.isfinite(v)], v[np.isfinite(v)]
    hi = ((bits.view(np.int32) >> 3).astype(np.int64) & 0x8FFFFFFF).astype(np.uint64)
    lo = (bits.astype(np.uint64) << np.uint64(29)) & np.uint64(0xFFFFFFFF)
    d = ((hi << np.uint64(32)) | lo).view(np.float64)
    want = v.astype(np.float64)
    assert np.array_equal(d * 2.0 ** 448 * 2.0 ** 448, want)
    assert np.array_equal(np.signbit(d), np.signbit(want))
    # a product and its scaled factor: the same bits as with the value itself
    w = rng.standard_normal(len(v))
    assert np.array_equal(d * (w * 2.0 ** 448) * 2.0 ** 448, want * w)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("precision", [16, 32, 64])
@pytest.mark.parametrize("persistent", [True, False])
def test_nonfinite_predictors_fail(bad, precision, persistent):
    x, y = W.latent_regression(8201, 70, 2, 4, 0.4, 3, dtype=np.float64)
    x[4000, 37] = bad
    xs = api.to_bf16(x.astype(np.float32)) if precision == 16 else x.astype(np.float32 if precision == 32 else np.float64)
    old = api.persistent()
    api.set_persistent(persistent)
    try:
        with pytest.raises(api._lib.FastplsError):
            api.fit_resident(np.asfortranarray(xs), y, ncomp=3, precision=precision)
    finally:
        api.set_persistent(old)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-40, 1e30])
def test_extreme_magnitudes(scale):
    """Subnormal and large FP32 predictors through the per-kernel loop: the FP64
    fit of the same values (R, Q and T scale out; 1e-6 for FP32 results)."""
    x, y = W.latent_regression(600, 90, 2, 4, 0.4, 8, dtype=np.float32)
    xs = (x.astype(np.float64) * scale).astype(np.float32)
    old = api.persistent()
    api.set_persistent(False)
    try:
        m32 = api.fit_resident(xs, y, ncomp=3, precision=32)
        m64 = api.fit_resident(xs.astype(np.float64), y.astype(np.float64), ncomp=3, precision=64)
        T32, T64 = m32.scores(), m64.scores()
        m32.close()
        m64.close()
    finally:
        api.set_persistent(old)
    assert np.max(np.abs(T32 - T64)) < 1e-6
