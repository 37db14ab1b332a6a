"""Whole rounds of the float64 block Jacobi in one launch (jb_pair_round_f64,
jb_worst_correlation_f64) against the general path of the same engine (batched
pair solves and GEMMs), at the edges of the kernel's forms: 8, 16 and 32
columns a pair, 32, 64, 96 and 128 rows, ragged last groups, wide input,
gradings and null columns."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = torch.finfo(torch.float64).eps


def _run(x, width, fused):
    S = importlib.import_module("pavel-s_svd_b200.solvers")
    BR = importlib.import_module("pavel-s_svd_b200.block_rounds")
    stats = {}
    pair, check, whole = S._pair_solver({}, stats)
    u, s, v = BR.raw(x, stats, {"block_size": width}, pair, check, S._complete_null_columns, whole if fused else None)
    return u, s, v, stats


@pytest.mark.parametrize("m,n,width", [
    (8, 5, 2), (32, 30, 4), (33, 11, 4), (64, 64, 4), (97, 17, 3), (128, 30, 4),       # up to 8 columns a pair
    (32, 32, 8), (33, 24, 8), (65, 40, 7), (96, 64, 8), (97, 50, 8), (128, 23, 6),     # up to 16
    (40, 40, 16), (64, 48, 16), (96, 70, 13), (128, 128, 16), (24, 96, 9),             # up to 32; wide
])
@pytest.mark.parametrize("kind", ["gaussian", "graded", "rank"])
def test_fused_rounds_are_the_general_rounds(m, n, width, kind):
    """Sigma within n eps sigma_1 a block sweep of the general path (each
    applies to a column at most n products of relative error eps), block
    sweeps within one, U and V orthonormal and U S V^H = A to the same bound."""
    g = torch.Generator(device="cuda").manual_seed(1000 * m + n)
    k = min(m, n)
    x = torch.randn(3, m, n, device="cuda", dtype=torch.float64, generator=g)
    if kind == "graded":
        x = x * torch.logspace(0, -8, n, device="cuda", dtype=torch.float64)
    if kind == "rank":
        r = max(1, k // 2)
        x = x[:, :, :r] @ torch.randn(3, r, n, device="cuda", dtype=torch.float64, generator=g)
        x = x / x.abs().amax()
    u, s, v, st = _run(x, width, True)
    _, s0, _, st0 = _run(x, width, False)
    tol = n * EPS * (st["block_sweeps"] + st0["block_sweeps"])
    assert abs(st["block_sweeps"] - st0["block_sweeps"]) <= 1
    assert float(((s - s0).abs().amax(-1) / s0[:, 0]).max()) <= tol
    eye = torch.eye(k, device="cuda", dtype=torch.float64)
    assert float((v.mT @ v - eye).abs().max()) <= 2 * k * tol
    # U of a column of relative size s_j / s_1 carries the column's error over s_j
    live = s[:, -1] > 1e-3 * s[:, 0]
    if bool(live.any()):
        assert float((u.mT @ u - eye).abs()[live].max()) <= 1e3 * tol
    rec = (u * s[:, None, :]) @ v.mT - x
    assert float((rec.norm(dim=(1, 2)) / x.norm(dim=(1, 2))).max()) <= k ** 0.5 * tol


@pytest.mark.parametrize("m,n", [(5, 3), (31, 31), (33, 33), (128, 65), (70, 64)])
def test_worst_correlation(m, n):
    """Against the torch form of the reference's test; a column of zeros and one
    below the live floor do not count."""
    N = importlib.import_module("pavel-s_svd_b200.native")
    g = torch.Generator(device="cuda").manual_seed(m + n)
    wt = torch.randn(4, n, m, device="cuda", dtype=torch.float64, generator=g)
    wt[1, n // 2] = 0
    wt[2, 0] = wt[2, 1] * 1e-20
    live = EPS * max(m, n)
    out = torch.empty(4 * n + 1, dtype=torch.float64, device="cuda")
    N.check(N.lib().jb_worst_correlation_f64(wt.data_ptr(), 4, m, n, live, out[1:].data_ptr(), out.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream), "jb_worst_correlation_f64")
    gm = wt @ wt.mT
    d = gm.diagonal(dim1=-2, dim2=-1)
    root = d.sqrt()
    keep = d > live ** 2 * d.amax(-1, keepdim=True)
    corr = gm.abs() / (root[:, :, None] * root[:, None, :]).clamp_min(torch.finfo(torch.float64).tiny)
    corr = torch.where(keep[:, :, None] & keep[:, None, :], corr, torch.zeros_like(corr))
    corr.diagonal(dim1=-2, dim2=-1).zero_()
    assert abs(float(out[0]) - float(corr.max())) <= 4 * m * EPS


def test_status_of_a_round():
    """Too few sweeps and a NaN are reported per pair, and the pair's columns left alone."""
    N = importlib.import_module("pavel-s_svd_b200.native")
    g = torch.Generator(device="cuda").manual_seed(3)
    wt = torch.randn(2, 8, 20, device="cuda", dtype=torch.float64, generator=g)
    wt[1, 5, 7] = float("nan")
    vt = torch.eye(8, device="cuda", dtype=torch.float64).expand(2, 8, 8).contiguous()
    before = wt.clone()
    cols = torch.tensor([[0, 1, 2, 3], [4, 5, 6, 7]], dtype=torch.int32, device="cuda")
    info = torch.full((2, 4), -1, dtype=torch.int32, device="cuda")

    def run(sweeps):
        N.check(N.lib().jb_pair_round_f64(wt.data_ptr(), vt.data_ptr(), cols.data_ptr(), 2, 20, 8, 2, 4, 0.0, sweeps,
                                          info[0].data_ptr(), info[1].data_ptr(),
                                          torch.cuda.current_stream().cuda_stream), "jb_pair_round_f64")
        return info[0].tolist()
    assert run(1) == [1, 1, 1, 2]
    assert torch.equal(wt.nan_to_num(7.0), before.nan_to_num(7.0))
    assert run(60) == [0, 0, 0, 2]
    assert torch.equal(wt[1, 4:].nan_to_num(7.0), before[1, 4:].nan_to_num(7.0))
    lib, p = N.lib(), wt.data_ptr()
    for bad in ((2, 129, 8, 2, 4), (2, 20, 8, 1, 33), (2, 20, 8, 2, 9)):
        b, m, n, k, c = bad
        n = max(n, c if c == 33 else n)
        m = max(m, n)
        with pytest.raises((RuntimeError, ValueError)):
            N.check(lib.jb_pair_round_f64(p, vt.data_ptr(), cols.data_ptr(), b, m, n, k, c, 0.0, 60,
                                          info[0].data_ptr(), info[1].data_ptr(), None), "jb_pair_round_f64")
