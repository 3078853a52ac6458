"""The FP32 MLP's activations and their derivatives (mlp_act, mlp_impl.cuh).

On the CPU: the polynomial of tanh in the source against tanh, and the fit
that gives such coefficients.  On the GPU: values and derivatives over both
signs, the split of tanh, large and non-finite arguments against FP64, and
against the same functions formed with torch's CUDA functions (expf, log1pf,
tanhf, sqrtf, IEEE division): no larger rms error."""
import ctypes
import re

import numpy as np
import pytest

from tmd_testutil import ROOT

SPLIT = 0.8  # |z| below which tanh is z + z^3 p(z^2)


def source_coefficients():
    txt = (ROOT / "lammps-tensormd_b200/csrc/mlp_impl.cuh").read_text()
    body = txt[txt.index("const float s = z * z;"):txt.index("const float y = mlp_select")]
    first = re.search(r"fmaf\((-?[\d.]+)f, s, (-?[\d.]+)f\)", body)
    rest = re.findall(r"fmaf\(p, s, (-?[\d.]+)f\)", body)
    assert f"mlp_select(t, {SPLIT}f, fmaf(t * s, p, t)" in txt
    return [np.float64(np.float32(c)) for c in [*first.groups(), *rest]][::-1]


def poly_error(c):
    """Largest relative error of t + t^3 p(t^2) below the split."""
    t = np.linspace(1e-3, SPLIT, 50001)
    return np.abs((t + sum(q * t ** (2 * k + 3) for k, q in enumerate(c))) / np.tanh(t) - 1).max()


def fit_tanh(terms):
    """Coefficients of p, each an FP32 number: least squares reweighted towards
    the smallest largest relative error (Lawson), one coefficient rounded at a
    time and the others fitted anew."""
    t = SPLIT * (1 - np.cos(np.pi * (np.arange(2000) + 0.5) / 2000)) / 2
    t = t[t > 1e-3]
    target, w = np.tanh(t) - t, 1 / np.tanh(t)
    basis = [t ** (2 * k + 3) for k in range(terms)]
    c = []
    for k in range(terms):
        rest = target - sum((q * b for q, b in zip(c, basis)), np.zeros_like(t))
        a = np.stack(basis[k:], 1)
        wt = w.copy()
        for _ in range(60):
            x = np.linalg.lstsq(a * wt[:, None], rest * wt, rcond=None)[0]
            e = np.abs((rest - a @ x) * w)
            wt *= np.sqrt(e / e.max() + 1e-3)
            wt /= wt.max()
        c.append(np.float64(np.float32(x[0])))
    return c


def test_tanh_polynomial():
    c = source_coefficients()
    assert len(c) == 6
    # an eighth of half an ulp, so that it does not show beside the rounding
    assert poly_error(c) < 2.0 ** -24 / 8
    # as good as the fit's own, up to the host's least-squares rounding
    assert poly_error(c) < 1.5 * poly_error(fit_tanh(6))
    assert poly_error(fit_tanh(5)) > 2.0 ** -25  # and one term less would show


def exact(actfn, z):
    z = z.astype(np.float64)
    if actfn == 1:
        return np.logaddexp(0.0, z), 1 / (1 + np.exp(-z))
    if actfn == 2:
        return np.tanh(z), 1 / np.cosh(z) ** 2
    q = np.sqrt(z * z + 4)
    y = np.where(z >= 0, 0.5 * (z + q), 2 / (q - z))
    return y, y / q


def with_cuda_functions(actfn, z):
    import torch
    z = torch.tensor(z, device="cuda")
    one, zero = torch.ones_like(z), torch.zeros_like(z)
    if actfn == 1:
        e = torch.exp(z)
        y, d = torch.where(z < 13.94, torch.log1p(e), z), one / (one + one / e)
    elif actfn == 2:
        e = torch.exp(-2 * z.abs())
        u = one + e
        y, d = torch.tanh(z), 4 * e / (u * u)
    else:
        q = torch.sqrt(torch.addcmul(zero + 4, z, z))
        y = torch.where(z >= 0, 0.5 * (z + q), 2 / (q - z))
        d = y / q
    return y.cpu().numpy(), d.cpu().numpy()


def on_device(actfn, z):
    from tmd_b200 import load_library
    z = np.ascontiguousarray(z, dtype=np.float32)
    y, d = np.empty_like(z), np.empty_like(z)
    p = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_float)) for a in (z, y, d)]
    assert load_library().tmd_mlp_activation(0, actfn, len(z), *p) == 0
    return y, d


# Largest relative errors in units of 2^-24 (half an ulp at worst), from the
# operations: expf within 2 ulp (4), log1pf 1 ulp (2), a reciprocal or square
# root from one Newton step 1.3, and 1 for every rounding of a result.
#   softplus: log1p's 2 and its argument's 4 (a factor a / ((1 + a) log1p a)
#   <= 1), the sum 1; derivative a / (1 + a): 4, 1.3, 1
#   tanh: far term (1 - T) / T <= 1/2 of 4 + 1.3 + 1, sum 1; derivative far:
#   4 (1 - a)/(1 + a) + 2 x 1.3 + 3, near: 2 T^2 / (1 - T^2) <= 1.6 of T's 2, 1
#   squareplus: q 1.3, the sum 1 (positive side), 2 / (q + |z|) 1.3 + 1.3;
#   derivative n / q: 2.6, 1.3, 1
BOUND = {1: (7, 6.3), 2: (4.2, 9.6), 3: (2.6, 4.9)}


@pytest.mark.gpu
@pytest.mark.parametrize("actfn", [1, 2, 3], ids=["softplus", "tanh", "squareplus"])
@pytest.mark.parametrize("top", [0.01, 1.0, 4.0, 12.0, 60.0])
def test_activation_accuracy(actfn, top):
    rng = np.random.default_rng(int(top * 100) + actfn)
    z = rng.uniform(-top, top, 1 << 20).astype(np.float32)
    if top == 1.0:  # every number around the split of tanh
        k = np.arange(-2000, 2000)
        near = (np.float32(SPLIT).view(np.int32) + k).astype(np.int32).view(np.float32)
        z[:8000] = np.concatenate([near, -near])
    for got, other, ref, bound in zip(on_device(actfn, z), with_cuda_functions(actfn, z),
                                      exact(actfn, z), BOUND[actfn]):
        use = np.abs(ref) > 1e-30  # normal FP32 numbers
        e = (got[use] - ref[use]) / ref[use]
        o = (other[use] - ref[use]) / ref[use]
        assert np.abs(e).max() <= bound * 2.0 ** -24
        # rms over 2^20 values: its own sampling noise is below 0.2%
        assert np.sqrt(np.mean(e * e)) <= 1.01 * np.sqrt(np.mean(o * o))


@pytest.mark.gpu
@pytest.mark.parametrize("actfn", [0, 1, 2, 3], ids=["relu", "softplus", "tanh", "squareplus"])
def test_activation_extremes(actfn):
    z = np.array([np.inf, -np.inf, np.nan, 3e38, -3e38, 1e20, -1e20, 1e15, -1e15, 1e9, -1e9,
                  200.0, -200.0, 0.0, -0.0, 1e-40, -1e-40], dtype=np.float32)
    y, d = on_device(actfn, z)
    with np.errstate(all="ignore"):
        if actfn == 0:  # a comparison: not-a-number counts as not positive
            ry, rd = np.where(z > 0, z, 0), (z > 0).astype(np.float32)
        else:
            ry, rd = exact(actfn, z)
    if actfn == 3:
        # z^2 overflows FP32 above 1.8e19: not finite there.  Values below
        # 1e-18 are held at that.
        big = (z > 1.8e19) | np.isnan(z)
        assert not np.isfinite(y[big]).any() and not np.isfinite(d[big]).any()
        y[big] = d[big] = ry[big] = rd[big] = 0.0
        ry, rd = np.maximum(ry, 1e-18), np.maximum(rd, 1e-36)
        y, d = np.maximum(y, 1e-18), np.maximum(d, 1e-36)
        ry[z == -np.inf], rd[z == -np.inf] = 1e-18, 1e-36
    if actfn == 1:
        rd[z == -np.inf] = 0.0
    assert np.allclose(y, ry, rtol=1e-6, atol=1e-37, equal_nan=True)
    assert np.allclose(d, rd, rtol=1e-6, atol=1e-37, equal_nan=True)
