"""The register eigen-solve of a block slot (jb_block_eig_f64_ex) against an FP64
simulation of the same odd-even sweep: scaled rotations with scales multiplied
back in during the sweep (dense G), tiles that cross lanes and warps in every
layout, zero and tiny columns."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sweeps(G, sweeps):
    """The kernel's sweeps in FP64: (Q, the smallest product of cosines a position saw)."""
    G = G.copy()
    n = G.shape[0]
    Q, scale, low = np.eye(n), np.ones(n), 1.0
    floor = np.finfo(np.float32).eps ** 2 * G.diagonal().max()
    for r in [r for _ in range(sweeps) for r in range(n)]:
        p = np.arange(r & 1, n - 1, 2)
        q = p + 1
        app, aqq, apq = G[p, p], G[q, q], G[p, q]
        on = (np.minimum(app, aqq) > floor) & (apq ** 2 > 1e-18 * app * aqq)
        z = np.where(on, abs(aqq - app) / (2 * np.where(apq == 0, 1, abs(apq))), 0)
        sign = np.where((aqq < app) != (apq < 0), -1, 1)         # equal diagonals: the sign of a_pq
        t = np.where(on, sign / (z + np.sqrt(1 + z * z)), 0)
        c = 1 / np.sqrt(1 + t * t)
        s = t * c
        for M in (G, Q):
            x, y = M[:, p].copy(), M[:, q].copy()
            M[:, p], M[:, q] = s * x + c * y, c * x - s * y
        x, y = G[p].copy(), G[q].copy()
        G[p], G[q] = s[:, None] * x + c[:, None] * y, c[:, None] * x - s[:, None] * y
        scale[p], scale[q] = c * scale[q], c * scale[p]
        low = min(low, scale.min())
    order = np.argsort(-G.diagonal(), kind="stable")
    return Q[:, order], G.diagonal()[order], low


def _dense(n, kind):
    rng = np.random.default_rng(n)
    if kind == "gaussian":
        x = rng.standard_normal((n, 2 * n))
        return x @ x.T / (2 * n)
    if kind == "signs":
        g = np.triu(np.sign(rng.standard_normal((n, n))), 1)
        return g + g.T + 2 * np.sqrt(n) * np.eye(n)
    x = rng.standard_normal((n, 2 * n)) * np.logspace(0, -5, n)[:, None]
    x[n // 3] = 0
    return x @ x.T / (2 * n)


@pytest.mark.parametrize("n", [64, 128])
@pytest.mark.parametrize("layout", [4, 8, 16])
@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("kind", ["gaussian", "signs", "graded"])
def test_one_sweep_is_the_simulated_one(n, layout, fp32, kind):
    """One sweep: Q orthogonal to n rotations of FP32 rounding, and what it
    leaves off the diagonal is the FP64 sweep's to n eps32 of |G| (a sweep
    applies n rounds, each of error eps32 relative to a column's norm)."""
    N = importlib.import_module("pavel-s_svd_b200.native")
    G = _dense(n, kind)
    q0, _, low = _sweeps(G.astype(np.float32).astype(np.float64), 1)
    if n == 128 and kind != "graded":
        assert low < 2.0 ** -8                       # the scales are multiplied in on the way
    g = torch.from_numpy(G).float().cuda()[None].contiguous()
    qt = [torch.empty(1, n, n, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    off, dmax = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
    sw = torch.zeros(1, dtype=torch.int32, device="cuda")
    N.check(N.lib().jb_block_eig_f64_ex(g.data_ptr(), qt[0].data_ptr(), qt[1].data_ptr(), qt[2].data_ptr(),
                                        off.data_ptr(), dmax.data_ptr(), sw.data_ptr(), 1, n, 1, 1e-9, None,
                                        layout | (N.EIG_FP32 if fp32 else 0),
                                        torch.cuda.current_stream().cuda_stream), "jb_block_eig_f64_ex")
    q = sum(x.double() for x in qt)[0].cpu().numpy().T
    eps = np.finfo(np.float32).eps
    assert np.abs(q.T @ q - np.eye(n)).max() <= n * eps
    g32 = g[0].double().cpu().numpy()

    def left(q):
        d = q.T @ g32 @ q
        return np.linalg.norm(d - np.diag(d.diagonal()))
    assert abs(left(q) - left(q0)) <= n * eps * np.linalg.norm(g32)
    ev = (q.T @ g32 @ q).diagonal()
    assert np.all(ev[:-1] >= ev[1:] - n * eps * abs(ev).max())
