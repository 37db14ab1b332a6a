"""The mixed solve by preconditioning and refinement (csrc/jb_mixed.cuh) and
its hand-over to the register kernels, against FP64 LAPACK and against the
register kernels themselves (the launch choice of 8-column blocks).

Tolerances, from the arithmetic: the refinement ends with every pair ratio of
W <= 10 eps32 (1.2e-6) and V orthogonal to 1e-8, in FP64; the outputs are
then rounded to FP32 (2^-24 relative).  So sigma agrees with LAPACK to 2^-24 +
n (1.2e-6)^2 relative (2e-7 taken), U is orthonormal to 1.2e-6 + 2^-23
(1.5e-6), V to 1e-8 + 2^-23 (2e-7), and A - U S Vh is below 3 * 2^-24 *
sqrt(n) sigma_1 (1.5e-6)."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def pkg():
    return importlib.import_module("pavel-s_svd_b200")


@pytest.fixture(scope="module")
def B():
    return importlib.import_module("pavel-s_svd_b200.batch")


def check(a, u, s, vh, values=None):
    a = np.asarray(a, np.float64)
    u, s, vh = (x.cpu().numpy().astype(np.float64) for x in (u, s, vh))
    k = s.shape[-1]
    truth = np.linalg.svd(a, compute_uv=False)[..., :k]
    top = truth[..., :1]
    assert float((np.abs(s - truth) / top).max()) <= 2e-7
    eye = np.eye(k)
    left, right = (1.5e-6, 2e-7) if a.shape[-2] >= a.shape[-1] else (2e-7, 1.5e-6)
    assert float(np.abs(np.swapaxes(u, -1, -2) @ u - eye).max()) <= left
    assert float(np.abs(vh @ np.swapaxes(vh, -1, -2) - eye).max()) <= right
    if k == min(a.shape[-2:]):
        assert float((np.abs(a - (u * s[..., None, :]) @ vh).max((-2, -1)) / top[..., 0]).max()) <= 1.5e-6


# both sides of every width class of the preconditioner (16, 32, 48, 64) and
# of the 8-wide tiles of the refinement; square, twice as tall, the tallest
SIZES = [(n, m) for n in (1, 2, 3, 8, 9, 16, 17, 32, 33, 40, 48, 49, 63, 64) for m in (n, min(2 * n + 1, 128), 128)]


@pytest.mark.parametrize("wide", [False, True], ids=["tall", "wide"])
@pytest.mark.parametrize("n,m", SIZES)
def test_sizes(pkg, n, m, wide):
    rng = np.random.default_rng(1000 * n + m)
    a = rng.standard_normal((3, m, n)).astype(np.float32)
    if wide:
        a = np.ascontiguousarray(np.swapaxes(a, 1, 2))
    check(a, *pkg.svd(torch.from_numpy(a).to(DEV)))


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e30])
@pytest.mark.parametrize("decades", [0.0, 3.0, 5.0, 8.0])
def test_spectra(pkg, decades, scale):
    """Equal values, graded ones, and ones the preconditioner hands over."""
    rng = np.random.default_rng(int(10 * decades))
    u, v = np.linalg.qr(rng.standard_normal((96, 50)))[0], np.linalg.qr(rng.standard_normal((50, 50)))[0]
    a = (((u * 10.0 ** (-decades * np.arange(50) / 49)) @ v.T) * scale).astype(np.float32)[None]
    check(a, *pkg.svd(torch.from_numpy(a).to(DEV)))


def test_output_forms(pkg):
    rng = np.random.default_rng(5)
    for shape in ((2, 60, 37), (2, 37, 60)):
        a = rng.standard_normal(shape).astype(np.float32)
        t = torch.from_numpy(a).to(DEV)
        u, s, vh = pkg.svd(t)
        ur, sr, vr = pkg.svd(t, rank=11)
        assert torch.equal(sr, s[:, :11]) and torch.equal(ur, u[:, :, :11]) and torch.equal(vr, vh[:, :11])
        none, sv, _ = pkg.svd(t, values_only=True)
        assert none is None and torch.equal(sv, s)
        uf, sf, vf = pkg.svd(t, full_matrices=True)
        assert uf.shape[-1] == shape[-2] and vf.shape[-2] == shape[-1]
        assert float((sf - s).abs().max()) <= 2e-7 * float(s.max())
        # strided input is the caller's: the same result as its copy
        assert torch.equal(pkg.svd(t.mT.contiguous().mT)[1], s)


def test_mixed_with_matrices_left_to_the_register_kernels(pkg, B):
    """One uneven batch of ordinary, rank-deficient, zero and graded matrices,
    in the default path and through the register kernels alone."""
    rng = np.random.default_rng(8)
    mats = [rng.standard_normal(s) for s in ((50, 40), (40, 50), (20, 9), (128, 64), (64, 64), (7, 7))]
    mats += [rng.standard_normal((60, 3)) @ rng.standard_normal((3, 45)), np.zeros((30, 12)), np.eye(33),
             np.ones((12, 40)), rng.standard_normal((64, 48)) * 10.0 ** (-7 * np.arange(48) / 47)]
    mats = [a.astype(np.float32) for a in mats]
    flat, m, n, off = B.pack(mats, DEV)
    plans = [B.UnevenBatch(m, n, DEV, a_off=off, launch=B.Launch(flags)) for flags in (0, pkg.native.BLOCK_WIDTH_8)]
    for plan in plans:
        plan.launch(flat)
        plan.check()
    for i, a in enumerate(mats):
        (u, s, vh), (_, s2, _) = plans[0].result(i), plans[1].result(i)
        assert float((s - s2).abs().max()) <= 2e-7 * max(float(s2[0]), 1e-30), i
        rec = (u.double() * s.double()) @ vh.double()
        assert float((rec.cpu() - torch.from_numpy(a).double()).abs().max()) <= 1.5e-6 * max(float(s[0]), 1e-30), i
        k = min(a.shape)
        eye = torch.eye(k, dtype=torch.float64, device=DEV)
        assert float((u.double().T @ u.double() - eye).abs().max()) <= 1.5e-6, i
        assert float((vh.double() @ vh.double().T - eye).abs().max()) <= 1.5e-6, i


def test_errors(pkg):
    a = torch.randn(3, 40, 24, device=DEV)
    with pytest.raises(RuntimeError, match="did not converge in 1 sweeps"):
        pkg.svd(a, max_sweeps=1)
    for bad in (float("nan"), float("inf"), float("-inf")):
        b = a.clone()
        b[1, 7, 5] = bad
        with pytest.raises(ValueError, match="NaN or infinity"):
            pkg.svd(b)
    assert bool(torch.isfinite(pkg.svd(a)[1]).all())


@pytest.mark.parametrize("n,m", [(1, 1), (8, 17), (16, 16), (17, 64), (20, 65), (24, 100), (31, 33), (32, 64), (32, 128)])
@pytest.mark.parametrize("wide", [False, True], ids=["tall", "wide"])
def test_large_batches_of_narrow_matrices(pkg, n, m, wide):
    """At most 32 columns in a batch of many matrices an SM: the refinement
    with half the threads, at the edges of its tiles; the same sums, so sigma is
    that of a batch of three to its rounding."""
    rng = np.random.default_rng(n + m)
    a = rng.standard_normal((1300, m, n)).astype(np.float32)
    if wide:
        a = np.ascontiguousarray(np.swapaxes(a, 1, 2))
    x = torch.from_numpy(a).to(DEV)
    u, s, vh = pkg.svd(x)
    pick = list(range(0, 1300, 61))
    check(a[pick], u[pick], s[pick], vh[pick])
    s3 = pkg.svd(x[610:613].contiguous())[1]
    assert float(((s[610:613] - s3).abs() / s3[:, :1]).max()) <= 2.0 ** -23


def test_uneven_width_classes(B):
    """An uneven batch of more than two matrices an SM: widths above and up to 32
    are refined by launches of their own; every matrix once."""
    rng = np.random.default_rng(12)
    n = rng.integers(1, 65, 700)
    m = np.minimum(n * rng.integers(1, 3, 700) + rng.integers(0, 3, 700), 128)
    m = np.maximum(m, n)
    plan = B.UnevenBatch(m, n, DEV)
    mats = [rng.standard_normal((int(p), int(q))).astype(np.float32) for p, q in zip(m, n)]
    flat = np.zeros(max(int(o) + t.size for t, o in zip(mats, plan.a_off)), np.float32)
    for t, o in zip(mats, plan.a_off):
        flat[int(o):int(o) + t.size] = t.ravel()
    plan.launch(torch.from_numpy(flat).to(DEV))
    torch.cuda.synchronize()
    assert int(plan.info[1].abs().max()) == 0
    for i in range(0, 700, 9):
        check(mats[i], *plan.result(i))
