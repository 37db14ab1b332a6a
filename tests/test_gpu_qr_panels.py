"""The Householder QR by row panels over a cluster of CTAs (qr_panel_kernel in
csrc/jb_qr.cu): every cluster size, shapes around its panel sizes, and the
kernels it leaves the largest matrices to.

Tolerances: n reflectors on m rows leave |QR - A| <= 50 m eps max|A| and |Q^H Q -
I| <= 50 m eps elementwise (as for the other QR tests); against the FP64 oracle
of the same reflectors R agrees to that bound too."""
import importlib

import numpy as np
import pytest
import torch

from oracle import jacobi_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
# (batch, m, n): one CTA (small, or a large batch), 2, 4, 8 and 16 CTAs, workspace
SHAPES = [(1, 1, 1), (3, 5, 5), (2, 31, 7), (300, 40, 9), (60, 130, 16), (30, 257, 33), (1, 300, 1), (1, 300, 64),
          (7, 513, 20), (1, 2048, 32), (1, 2047, 31), (1, 4096, 60), (1, 4000, 90)]


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_panels(shape, dt):
    Q = importlib.import_module("pavel-s_svd_b200.qr")
    rng = np.random.default_rng(sum(shape))
    a = rng.standard_normal(shape)
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal(shape)
    a = a.astype(dt)
    if shape[-1] > 4:
        a[0, :, 2] = 0                      # a zero column: no reflector
        a[-1, :, 3] = a[-1, :, 1]           # a dependent one
    q, r = (x.cpu().numpy().astype(np.complex128) for x in Q.qr(torch.from_numpy(a).to(DEV)))
    m, n = shape[-2:]
    tol = 50 * m * float(np.finfo(dt).eps)
    top = max(1.0, float(np.abs(a).max()))
    assert np.array_equal(r, np.triu(r))
    assert float(np.abs(q @ r - a).max()) <= tol * top
    assert float(np.abs(np.conj(np.swapaxes(q, 1, 2)) @ q - np.eye(n)).max()) <= tol
    if n <= 4:
        qo, ro = O.qr(a.astype(np.complex128 if np.iscomplexobj(a) else np.float64))
        assert float(np.abs(r - ro).max()) <= tol * top and float(np.abs(q - qo).max()) <= tol


@pytest.mark.parametrize("scale", [1e-200, 1e-160, 1e160, 1e200])
def test_range(scale):
    """Entries whose squares leave the range: a diagonal matrix (only alpha is
    large) in FP64, where the norm comes from hypot."""
    Q = importlib.import_module("pavel-s_svd_b200.qr")
    a = np.diag(np.arange(1.0, 9.0))[None] * scale
    q, r = (x.cpu().numpy() for x in Q.qr(torch.from_numpy(a).to(DEV)))
    assert float(np.abs(q @ (r / scale) - a / scale).max()) <= 1e-13 and np.isfinite(r).all()
