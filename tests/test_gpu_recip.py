"""The reciprocals, inverse square roots and quotients of csrc/recip.cuh against 80-bit arithmetic
on the CPU and against CUDA's own functions, over the ranges that their comments state.

The bars are the error bounds derived there, in units of the last place's half (u = 2^-53 or
2^-24): one rounding of the last operation, the series' rest for an approximation off by less than
2^-18, and the rounding of x y in the inverse square root.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
N = 1 << 21


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    from bem3d_elastostatic_b200 import build

    so = str(tmp_path_factory.mktemp("recip") / "probe.so")
    subprocess.run([build.NVCC, *build.ARCH, *build.COMMON, "-I", build.CSRC, "-shared", "-o", so,
                    os.path.join(HERE, "recip_probe.cu"), "-lcudart"], check=True)
    return ctypes.CDLL(so)


def _call(fn, x, v, rows):
    import torch

    xd, vd = torch.as_tensor(x, device="cuda"), torch.as_tensor(v, device="cuda")
    out = torch.empty((rows, x.size), dtype=xd.dtype, device="cuda")
    torch.cuda.synchronize()
    assert fn(x.size, *(ctypes.c_void_p(t.data_ptr()) for t in (xd, vd, out))) == 0
    return out.cpu().numpy()


def _spread(rng, lo, hi, n):
    """Positive numbers with exponents uniform in [lo, hi), a quarter of them next to 1."""
    x = np.ldexp(1.0 + rng.random(n), rng.integers(lo, hi, n))
    x[: n // 4] = 4.0 ** rng.uniform(0.0, 1.0, n // 4)
    return x


def _rel(got, exact):
    return float(np.abs(got.astype(np.longdouble) / exact - 1).max())


def test_inverse_square_root(probe):
    rng = np.random.default_rng(0)
    x = _spread(rng, -1022, 1023, N)
    x[-6:] = [2.0 ** -1022, 2.0 ** 1022, 1.0, np.nextafter(1.0, 0), np.nextafter(4.0, 0), np.finfo(float).max]
    o = _call(probe.probe_fp64, x, x, 7)
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    e = float(np.abs(1 - x.astype(np.longdouble) * o[0].astype(np.longdouble) ** 2).max())
    u = 2.0 ** -53
    print(f"rsqrt: approximation 2^{np.log2(e):.2f}, error {_rel(o[1], exact) / u:.3f} u, CUDA {_rel(o[2], exact) / u:.3f} u")
    assert e < 2.0 ** -18
    assert _rel(o[1], exact) <= 1.7 * u
    assert (np.abs(o[1] - o[2]) <= 2 * np.spacing(o[2])).all()  # 1.7 u and CUDA's 1 ulp, on the same grid


def test_reciprocal_and_quotient(probe):
    rng = np.random.default_rng(1)
    x = _spread(rng, -963, 963, N)  # 1e-290 .. 1e290
    x[1::2] *= -1.0
    v = x * rng.uniform(-1.0, 1.0, N)  # a multiplier's numerator
    v[np.abs(v) < 1e-270] = 0.0
    o = _call(probe.probe_fp64, x, v, 7)
    xl, u = x.astype(np.longdouble), 2.0 ** -53
    e = float(np.abs(1 - xl * o[3].astype(np.longdouble)).max())
    nz = v != 0
    q = v.astype(np.longdouble)[nz] / xl[nz]
    print(f"reciprocal: approximation 2^{np.log2(e):.2f}, error {_rel(o[4], 1 / xl) / u:.3f} u; "
          f"quotient {_rel(o[5][nz], q) / u:.5f} u, other than CUDA's {np.mean(o[5] != o[6]):.2g}")
    assert e < 2.0 ** -18
    assert _rel(o[4], 1 / xl) <= 1.6 * u
    assert _rel(o[5][nz], q) <= (1 + 2.0 ** -10) * u
    assert (o[5][~nz] == 0).all()
    assert (np.abs(o[5] - o[6]) <= np.spacing(np.abs(o[6]))).all()


def test_fp32(probe):
    rng = np.random.default_rng(2)
    x = _spread(rng, -99, 99, N).astype(np.float32)  # 1e-30 .. 1e30
    x[1::2] *= -1
    v = (x * rng.uniform(-1.0, 1.0, N)).astype(np.float32)
    v[np.abs(v) < 1e-29] = 0
    o = _call(probe.probe_fp32, x, v, 5)
    xl, u, nz = x.astype(np.longdouble), 2.0 ** -24, v != 0
    q = v.astype(np.longdouble)[nz] / xl[nz]
    print(f"fp32: reciprocal {_rel(o[0], 1 / xl) / u:.4f} u; quotients {_rel(o[1][nz], q) / u:.5f}, "
          f"{_rel(o[4][nz], q) / u:.5f} u, other than CUDA's {np.mean(o[1] != o[2]):.2g}")
    assert _rel(o[0], 1 / xl) <= 1.01 * u
    for k in (1, 4):
        assert _rel(o[k][nz], q) <= (1 + 2.0 ** -10) * u
        assert (np.abs(o[k] - o[2]) <= np.spacing(np.abs(o[2]))).all()
