"""Arithmetic that stands for divisions in the kernels, on the device against
the divisions, value for value (tests/arithmetic_harness.cu)."""

from __future__ import annotations

import ctypes
from pathlib import Path
import subprocess

import numpy as np
import pytest

from ordinarylight_b200 import build

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def harness(tmp_path_factory, cuda_device):
    out = tmp_path_factory.mktemp("arithmetic") / "libarithmetic.so"
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", "-I", str(build.INCLUDE), "-I", str(build.CSRC),
                    str(HERE / "arithmetic_harness.cu"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


def _shear(harness, d):
    import torch

    x = torch.as_tensor(np.ascontiguousarray(d, np.float32), device="cuda")
    got, want = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(a.data_ptr()) for a in (x, got, want)]
    assert harness.shear_terms(ctypes.c_uint32(len(d)), *p) == 0
    return got.cpu().numpy(), want.cpu().numpy()


def _same(got, want):
    """The same value (a zero's sign does not matter to the hit test) or both undefined."""
    return (got == want) | (np.isnan(got) & np.isnan(want))


def test_shear_terms_are_the_rounded_quotients(harness):
    """Directions of every length a float32 holds, with components between 1
    and 2^-60 of the largest, and random and extreme mantissas."""
    rng = np.random.default_rng(8)
    n = 4_000_000
    mantissa = rng.integers(0, 1 << 23, (n, 3), dtype=np.uint32)
    mantissa[::5] = rng.choice(np.uint32([0, 1, 2, (1 << 23) - 1, (1 << 23) - 2, 1 << 22]), (len(mantissa[::5]), 3))
    top = rng.integers(-40, 60, (n, 1))
    exponent = top - rng.integers(0, 61, (n, 3))
    exponent[np.arange(n), rng.integers(0, 3, n)] = top[:, 0]
    sign = rng.integers(0, 2, (n, 3)).astype(np.uint32) << np.uint32(31)
    d = (sign | ((exponent + 127).astype(np.uint32) << np.uint32(23)) | mantissa).view(np.float32)
    got, want = _shear(harness, d)
    assert _same(got, want).all()


def test_shear_terms_of_extreme_directions(harness):
    """Zero, subnormal, huge and infinite components: the divisions' values,
    whatever those are.  (With an undefined component no triangle is hit.)"""
    edge = np.float32([0.0, 1e-45, 1e-39, 1e-38, 2e-38, 1e-31, 9.9e-21, 1e-20, 1.1e-20, 9.9e-19, 1.1e-18, 1.0,
                       9.9e17, 1.1e18, 1e30, 1e38, 3.4e38, np.inf])
    edge = np.concatenate([edge, -edge])
    d = np.stack(np.meshgrid(edge, edge, edge), -1).reshape(-1, 3)
    got, want = _shear(harness, d)
    top = np.abs(d).max(1, keepdims=True)
    same = _same(got, want)
    assert same[:, 2].all()
    # of a component below 2^-100 the residual may lie under the smallest subnormal: the correction may be one step off
    with np.errstate(invalid="ignore"):   # 0 * inf
        tiny = (np.abs(want[:, :2] * top) < 2.0 ** -100) & (top < 1e18) & (top > 1e-18)
    assert (same[:, :2] | tiny).all()
    off = np.abs(got[:, :2].astype(np.float64) - want[:, :2])
    assert (off[tiny] <= np.spacing(np.abs(want[:, :2][tiny]))).all()


def test_byte_texels_are_the_rounded_quotients(harness):
    import torch

    got, want = torch.empty(256, device="cuda"), torch.empty(256, device="cuda")
    torch.cuda.synchronize()
    assert harness.byte_texels(ctypes.c_void_p(got.data_ptr()), ctypes.c_void_p(want.data_ptr())) == 0
    assert torch.equal(got, want)
    np.testing.assert_array_equal(want.cpu().numpy(), np.arange(256, dtype=np.float32) / np.float32(255.0))
