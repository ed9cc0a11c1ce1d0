"""The FP64 adjoint's own reciprocal and square root (p2r_math_check64) against the correctly rounded
1 / b and sqrt(x) of the host, bit for bit: over the exponents of the path and far beyond, with random
mantissas and with those around the powers of two, where the rounding is hardest. A divisor with all
mantissa bits set is the one exception, one unit lower; its reciprocal lies 2^-54 of a unit above the
middle of two doubles."""
import numpy as np
import pytest

N = 1 << 21
ALL_ONES = np.uint64((1 << 52) - 1)


def doubles(rng, lo, hi, mantissas):
    """N positive doubles in [2^lo, 2^(hi+1))."""
    m = rng.integers(0, 1 << 52, N, dtype=np.uint64)
    if mantissas == "edges":  # k 0s or 1s, then random bits
        m >>= rng.integers(0, 53, N, dtype=np.uint64)
        m = np.where(rng.integers(0, 2, N) == 1, ALL_ONES - m, m)
    e = rng.integers(1023 + lo, 1023 + hi + 1, N).astype(np.uint64)
    return ((e << np.uint64(52)) | m).view(np.float64)


def on_gpu(a):
    import torch

    import p2r_tests_b200 as p2r
    inv, root = p2r.math_check64(torch.from_numpy(a).cuda())
    torch.cuda.synchronize()
    return inv.cpu().numpy(), root.cpu().numpy()


def bits(a):
    return a.view(np.int64)


@pytest.mark.gpu
@pytest.mark.parametrize("mantissas", ["random", "edges"])
@pytest.mark.parametrize("lo,hi", [(-20, 19), (-900, 900)])
def test_rounded_as_the_language_has_them(lo, hi, mantissas):
    x = doubles(np.random.default_rng(lo * lo + len(mantissas)), lo, hi, mantissas)
    inv, root = on_gpu(x)
    lower = (x.view(np.uint64) & ALL_ONES) == ALL_ONES
    assert lower.any() == (mantissas == "edges")
    assert np.array_equal(bits(inv), bits(1.0 / x) - lower)
    assert np.array_equal(bits(root), bits(np.sqrt(x)))
    neg, _ = on_gpu(-x)
    assert np.array_equal(bits(neg), bits(-inv))


@pytest.mark.gpu
def test_whole_range_of_normal_numbers():
    x = doubles(np.random.default_rng(3), -1022, 1022, "edges")
    inv, root = on_gpu(x)
    normal = x < 2.0 ** 1021  # the reciprocal is a normal number
    assert (np.abs(bits(inv) - bits(1.0 / x))[normal] <= 1).all()
    assert (np.abs(bits(root) - bits(np.sqrt(x))) <= 1).all()


@pytest.mark.gpu
def test_special_arguments():
    with np.errstate(divide="ignore"):
        a = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, -1e-310, 1.7e308])
        inv, root = on_gpu(a)
        assert np.array_equal(bits(inv[:4]), bits(1.0 / a[:4])) and np.isnan(inv[4])
    assert np.array_equal(inv[5:7], [np.inf, -np.inf]) and inv[7] == 0.0  # subnormals count as 0
    assert np.array_equal(bits(root[:3]), bits(a[:3])) and np.isnan(root[4])
    assert root[5] == 1e-310 and root[7] == np.sqrt(1.7e308)


def test_bad_arguments_are_refused():
    import p2r_tests_b200 as p2r
    lib = p2r.lib()
    assert lib.p2r_math_check64(-1, None, None, None, None) == 1
    assert lib.p2r_math_check64(4, None, None, None, None) == 1
    assert lib.p2r_math_check64(0, None, None, None, None) == 0
