"""rcp_f64, sqrt_f64, cut_f32 and the float pairs against CUDA's division, root and
conversions, and root_n against the root in extended precision, over random
mantissas of every exponent and the edges of their guards.

Tolerances: with a residual e < 2^-18 of the first approximation, the truncated
series of 1/(1 - e) errs by e^3 < 2^-54 and that of 1/sqrt(1 - e) by 5/16 e^3;
with the last rounding (and half of that of x y, for the root) each lies within
one ulp of the correctly rounded value.  root_n: its two sums, the reciprocal, two
products and the power of the start value round by some 2^-53 each, and Halley's
step leaves (n^2 - 1)/12 e^3 < 2^-55 of a start value good to 4e-6: below 8 ulp.
Outside its guard exp2(log2(x) / n): an ulp of a logarithm of 106 over n, half an ulp
of the quotient and the rounding of 1/n, times ln 2: below 120 ulp."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests import device_math

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib(cuda):
    return device_math.load()


def call(lib, name, x, width, dtype=torch.float64, *args):
    xd = torch.tensor(x, device="cuda")
    out = torch.zeros(width * len(x), dtype=dtype, device="cuda")
    torch.cuda.synchronize()
    assert getattr(lib, name)(len(x), *args, device_math.ptr(xd), device_math.ptr(out)) == 0
    return out.cpu().numpy().reshape(width, -1)


def numbers():
    """Every exponent with 400 mantissas, their edges, and the special values."""
    rng = np.random.default_rng(91)
    ex = np.repeat(np.arange(2047, dtype=np.uint64), 406)
    man = rng.integers(0, 1 << 52, ex.size, dtype=np.uint64)
    edge = np.array([0, 1, (1 << 52) - 1, (1 << 52) - 2, 1 << 51, 1 << 32], np.uint64)
    man.reshape(2047, 406)[:, :6] = edge
    x = ((ex << np.uint64(52)) | man).view(np.float64)
    return np.concatenate([x, -x, [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324]])


def ulps(a, b):
    """|a - b| in units of b's last place; equal values, infinities and NaN count 0."""
    same = (a == b) | (np.isnan(a) & np.isnan(b))
    with np.errstate(invalid="ignore", over="ignore"):
        d = np.abs(a - b) / np.spacing(np.abs(b))
    return np.where(same, 0.0, np.where(np.isnan(d), np.inf, d))


def test_reciprocal_and_root(cuda, lib):
    r, r_ref, s, s_ref = call(lib, "check_roots", numbers(), 4)
    assert ulps(r, r_ref).max() <= 1.0
    assert ulps(s, s_ref).max() <= 1.0


@pytest.mark.parametrize("n", [2, 3, 4, 5, 7, 10, 16])
def test_root_n(cuda, lib, n):
    rng = np.random.default_rng(92)
    x = np.concatenate([10.0 ** rng.uniform(-32, 32, 200000), 1.0 + rng.uniform(-1e-3, 1e-3, 50000), [1.0, 1e-30, 1e30]])
    (r,) = call(lib, "check_root_n", x, 1, torch.float64, n, C.c_double(1.0 / n))
    ref = (x.astype(np.longdouble) ** (np.longdouble(1) / n)).astype(np.float64)
    assert ulps(r, ref)[np.abs(np.log10(x)) < 29.9].max() <= 8.0
    assert ulps(r, ref).max() <= 120.0


def test_cut_to_fp32(cuda, lib):
    a, b = call(lib, "check_cut", numbers(), 2, torch.int32)
    x = numbers()
    assert np.array_equal(a[~np.isnan(x)], b[~np.isnan(x)])
    assert np.isnan(a[np.isnan(x)].view(np.float32)).all()


def test_float_pair_split_and_join(cuda, lib):
    """hi = float(x), lo = float(x - hi) by bit operations, and back, also outside
    their exponent range and at the carry into the next power of two."""
    a = call(lib, "check_split", numbers(), 4, torch.int32)
    x = numbers()
    ok = ~np.isnan(x)
    assert np.array_equal(a[0][ok], a[2][ok])
    fin = ok & np.isfinite(a[2].view(np.float32))
    assert np.array_equal(a[1][fin].view(np.float32), a[3][fin].view(np.float32))  # (a zero's sign may differ)
    f = np.concatenate([a[2][fin], a[3][fin]]).view(np.float32)
    with np.errstate(invalid="ignore"):
        w = call(lib, "check_widen", f, 1)[0]
    tiny = np.abs(f) < np.finfo(np.float32).tiny  # flushed or not, as the conversion does
    assert np.array_equal(w[~tiny], f[~tiny].astype(np.float64))
