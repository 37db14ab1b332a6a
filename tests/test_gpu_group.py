"""The sweeps with several lanes a block pair (csrc/jb_group.cuh): float64, plain
FP32, complex64 and complex128 on both sides of every register-tile size,
against FP64 LAPACK.

Tolerances, from the arithmetic: a column takes at most 12 sweeps x 64
rotations, each rounding its elements to eps / 2, so W and V end about
sqrt(768) eps off in norm and direction: 3.3e-6 (FP32), 6e-15 (FP64).
Columns of W are left with pair ratios <= 10 eps.  Taken: 1e-5 and 5e-14 for
sigma and the reconstruction (of sigma_1) and for the orthonormality of U and
V; a column of U of a small sigma is as orthogonal as the others, as the
active test is relative."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
# (m, n): edges of the tiles (16, 32, 64 columns; 32, 48, 64, 128 rows), odd sizes
SIZES = [(1, 1), (2, 2), (5, 3), (32, 16), (31, 15), (33, 16), (128, 16), (96, 13), (17, 17), (48, 17), (48, 32),
         (49, 32), (64, 32), (64, 31), (65, 32), (128, 32), (33, 33), (64, 33), (64, 64), (65, 64), (100, 47), (128, 64),
         (32, 32), (30, 24), (47, 16), (60, 14), (64, 16), (65, 16), (96, 32), (97, 30), (60, 40), (96, 64), (97, 50)]


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("pavel-s_svd_b200")


def bound(dt):
    return 1e-5 if dt in (np.float32, np.complex64) else 5e-14


def check(a, u, s, vh):
    dt = a.dtype.type
    wide = np.complex128 if np.iscomplexobj(a) else np.float64
    u, s, vh = (x.resolve_conj().cpu().numpy() for x in (u, s, vh))
    u, vh, s, a = u.astype(wide), vh.astype(wide), s.astype(np.float64), a.astype(wide)
    r = s.shape[-1]
    truth = np.linalg.svd(a, compute_uv=False)
    top = truth[..., :1]
    assert float((np.abs(s - truth) / top).max()) <= bound(dt)
    assert float(np.abs(np.conj(np.swapaxes(u, -1, -2)) @ u - np.eye(u.shape[-1])).max()) <= bound(dt)
    assert float(np.abs(vh @ np.conj(np.swapaxes(vh, -1, -2)) - np.eye(vh.shape[-2])).max()) <= bound(dt)
    rec = (u[..., :r] * s[..., None, :]) @ vh[..., :r, :]
    assert float((np.abs(rec - a).max((-2, -1)) / top[..., 0]).max()) <= bound(dt)


def matrices(shape, dt, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal(shape)
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal(shape)
    return a.astype(dt)


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("m,n", SIZES)
def test_sizes(pkg, m, n, dt):
    for shape in ((3, m, n), (2, n, m)):
        a = matrices(shape, dt, 100 * m + n)
        check(a, *pkg.svd(torch.from_numpy(a).to(DEV), precision="fp32"))


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
def test_graded_deficient_and_full(pkg, dt):
    """Columns over 12 decades of scale, a rank-deficient matrix and a zero one
    in a batch, full bases at the widest register tile."""
    rng = np.random.default_rng(3)
    a = matrices((3, 60, 30), dt, 4)
    a[0] *= (10.0 ** (-12 * rng.random(30))).astype(np.float32)
    a[1, :, 5:] = a[1, :, :1]
    a[2] = 0
    u, s, vh = pkg.svd(torch.from_numpy(a).to(DEV), precision="fp32")
    eye = np.eye(30)
    un, vn = u.resolve_conj().cpu().numpy(), vh.resolve_conj().cpu().numpy()
    for z in range(3):
        assert float(np.abs(np.conj(un[z].T) @ un[z] - eye).max()) <= 2 * bound(dt)
        rec = (un[z].astype(np.complex128) * s[z].cpu().numpy()) @ vn[z]
        assert float(np.abs(rec - a[z]).max()) <= bound(dt) * max(float(s[z].max()), 1e-30)
    assert float(s[2].max()) == 0
    b = matrices((1, 128, 60), dt, 5)
    uf, sf, vf = pkg.svd(torch.from_numpy(b).to(DEV), precision="fp32", full_matrices=True)
    assert uf.shape[-1] == 128
    check(b, uf, sf, vf)


def test_uneven_equals_equal_shapes(pkg):
    """A matrix of an uneven FP32 batch, in either size class, is solved with
    the same sums as in a batch of its own shape."""
    B = importlib.import_module("pavel-s_svd_b200.batch")
    mats = [matrices(s, np.float32, i) for i, s in enumerate([(40, 33), (64, 64), (65, 40), (128, 64), (20, 9), (30, 70),
                                                              (100, 31), (33, 32), (1, 1), (7, 120)])]
    flat, m, n, off = B.pack(mats, DEV)
    plan = B.UnevenBatch(m, n, DEV, a_off=off, precision="fp32")
    plan.launch(flat)
    plan.check()
    for i, a in enumerate(mats):
        u, s, vh = pkg.svd(torch.from_numpy(a).to(DEV), precision="fp32")
        for x, y in zip(plan.result(i), (u, s, vh)):
            assert torch.equal(x, y), i


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 31, 32, 33, 63, 64, 65])
def test_eigen_sizes(n, dt):
    """The two-sided solve on the same sweeps, both sides of its sizes (16, 32,
    64; 65 is the shared-memory kernel): indefinite, zero-diagonal (max|H| off
    the diagonal) and zero matrices in one batch.  Eigenvalues to 10 n eps
    max|w|, V and the residual to 100 n eps (n rotations a sweep, 10 sweeps)."""
    E = importlib.import_module("pavel-s_svd_b200.eigh")
    x = matrices((3, n, n), dt, n)
    h = x + np.conj(np.swapaxes(x, 1, 2))
    h[1] = 0
    h[1][np.arange(n - 1), np.arange(1, n)] = 1
    h[1][np.arange(1, n), np.arange(n - 1)] = 1
    h[2] = 0
    w, v, sweeps = E.jacobi_eigh(torch.from_numpy(h).to(DEV))
    w, v = w.cpu().numpy().astype(np.float64), v.resolve_conj().cpu().numpy().astype(np.complex128)
    eps = float(np.finfo(dt).eps)
    truth = np.linalg.eigvalsh(h.astype(np.complex128))
    scale = np.maximum(np.abs(truth).max(-1), 1e-300)
    assert sweeps >= 1 and float((np.abs(w - truth).max(-1) / scale).max()) <= 10 * n * eps
    assert float(np.abs(np.conj(np.swapaxes(v, 1, 2)) @ v - np.eye(n)).max()) <= 100 * n * eps
    res = np.abs(h.astype(np.complex128) @ v - v * w[:, None, :]).max((-2, -1)) / scale
    assert float(res.max()) <= 100 * n * eps


@pytest.mark.parametrize("dt", [np.float32, np.complex64, np.complex128])
@pytest.mark.parametrize("m,n", [(60, 16), (100, 16), (33, 9)])
def test_large_batches_take_the_same_sums(pkg, m, n, dt):
    """Up to 16 columns a large batch has half the threads a matrix: the same
    lanes a pair, so sigma of a matrix is the same to the last rounding of its
    norm (2 eps sigma_1) as in a batch of three."""
    a = matrices((700, m, n), dt, m + n)
    x = torch.from_numpy(a).to(DEV)
    s = pkg.svd(x, precision="fp32")[1]
    for k in (0, 350, 697):
        u3, s3, v3 = pkg.svd(x[k:k + 3].contiguous(), precision="fp32")
        assert float((s[k:k + 3] - s3).abs().max()) <= 2 * torch.finfo(s.dtype).eps * float(s3.max())
        check(a[k:k + 3], u3, s3, v3)
    u, s, vh = pkg.svd(x[:400].contiguous(), precision="fp32")
    check(a[:400], u, s, vh)
