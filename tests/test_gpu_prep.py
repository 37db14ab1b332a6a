"""jb_prepare and jb_check_finite (csrc/jb_prep.cu): scaling by a power of two,
transposition, widening, the input and output checks.  The scaled values are
exact, so they are compared bit for bit."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def S():
    return importlib.import_module("pavel-s_svd_b200.solvers")


@pytest.mark.parametrize("dt", [torch.float32, torch.float64, torch.complex64, torch.complex128])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 31, 33), (2, 32, 64), (5, 1, 70), (1, 300, 5), (70000, 2, 1)])
def test_prepare(S, dt, shape):
    rng = np.random.default_rng(7)
    a = rng.standard_normal(shape) * 10.0 ** rng.integers(-30, 30, size=(shape[0], 1, 1))
    if dt.is_complex:
        a = a + 1j * a[..., ::-1]
    a[0] = 0
    t = torch.from_numpy(a).to(dt).to(DEV)
    forms = [t, t.mT.contiguous().mT, torch.cat([t, t], -1)[..., :shape[-1]]]     # strides are the caller's
    if dt.is_complex:
        forms += [t.conj().resolve_conj().conj()]                                 # a lazy conjugate
    top = torch.view_as_real(t).abs().amax(-1) if dt.is_complex else t.abs()
    expo = torch.frexp(top.double().amax((1, 2)))[1]
    for x in forms:
        for transpose in (False, True):
            out, scale, words = S._prepare(x, transpose)
            assert words.read() == 0
            assert torch.equal(scale, torch.ldexp(torch.ones_like(scale), expo))
            ref = t.mH if transpose else t
            want = torch.stack([r / s for r, s in zip(ref[:50], scale[:50].to(t.real.dtype))])
            assert torch.equal(out[:50], want.resolve_conj()) and out.is_contiguous()
            assert torch.equal(out * scale.to(t.real.dtype)[:, None, None], ref.resolve_conj())
    if dt == torch.float32:
        out, scale, words = S._prepare(t, False, widen=True)
        assert out.dtype == torch.float64 and torch.equal(out * scale[:, None, None], t.double())


@pytest.mark.parametrize("dt", [torch.float32, torch.float64, torch.complex64, torch.complex128])
def test_checks(S, dt):
    x = torch.randn(4, 37, 21, dtype=dt, device=DEV)
    for bad in (float("nan"), float("inf"), float("-inf")):
        y = x.clone()
        y[2, 36, 20] = bad
        _, _, words = S._prepare(y, True)
        with pytest.raises(ValueError, match="NaN or infinity"):
            words.read()
        for z in (y, y.mT, y[:, 1:, ::2]):
            words = S._Verdicts(4, DEV)
            words.check_finite(x, z)
            with pytest.raises(RuntimeError, match="nonfinite output"):
                words.read()
    words = S._Verdicts(4, DEV)
    words.check_finite(x, x.mT, x[:, 3:], x[:0])
    assert words.read() == 0


@pytest.mark.parametrize("alg", ["jacobi", "gram_jacobi", "qr", "tsqr", "randomized", "block_jacobi"])
def test_nan_in_one_matrix_of_a_batch(alg):
    """The input check comes before any other error, whatever the solver does
    with the other matrices."""
    pkg = importlib.import_module("pavel-s_svd_b200")
    for dt in (torch.float32, torch.float64, torch.complex64):
        for shape in ((3, 300, 12), (3, 40, 24)):
            for bad in (float("nan"), float("inf")):
                x = torch.randn(*shape, dtype=dt, device=DEV)
                x[1, 5, 7] = bad
                with pytest.raises(ValueError, match="NaN or infinity"):
                    pkg.svd(x, alg, block_size=4, rank=6)
