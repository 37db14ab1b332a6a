"""The blocked null completion at the edges of its layout: one to 64 published
rows a CTA (one-warp selection or sort), more rows than the candidate set
takes, CTAs of more than one 64-row pass, ragged last steps of the row products
(odd column counts, FP32 and FP64 rows), a last block of a few columns."""
import importlib

import numpy as np
import pytest
import torch

from oracle import jacobi_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,n,kept", [
    (319, 206, 61),        # 4 CTAs, 64 rows published by each (sorted)
    (1023, 129, 30),       # 15 CTAs of up to 69 rows, 17 published (sorted)
    (1100, 67, 1),         # 17 CTAs, 15 published (one warp)
    (8190, 45, 3),         # 127 CTAs, two published: 254 for 128 candidates
    (9600, 39, 5),         # every SM one row
    (40000, 35, 2),        # more than 256 rows a CTA: the sort again
])
def test_pivots_and_columns_are_the_per_column_algorithms(dtype, m, n, kept):
    """Against the oracle in FP64.  Bounds: eps times the columns built on one
    another (<= 200) times a leverage's growth 1 / (1/2) per column's length,
    with the FP32 rows rounded once a column: 1e-11 and 5e-5."""
    S = importlib.import_module("pavel-s_svd_b200.solvers")
    rng = np.random.default_rng(m + n)
    q = np.linalg.qr(rng.standard_normal((m, kept)))[0]
    keep = np.zeros((1, n), bool)
    keep[0, rng.choice(n, kept, replace=False)] = True
    u = rng.standard_normal((1, m, n))
    u[0][:, keep[0]] = q
    u = u.astype(dtype)
    want = O.complete_null_columns(u.astype(np.float64), keep)
    got = S._complete_null_columns(torch.from_numpy(u).cuda(), torch.from_numpy(keep).cuda()).cpu().numpy()
    miss = ~keep[0]
    assert np.array_equal(np.abs(got[0][:, miss]).argmax(0), np.abs(want[0][:, miss]).argmax(0))
    err = np.abs(got.astype(np.float64) - want).max()
    assert err <= (1e-11 if dtype == np.float64 else 5e-5), err
    g64 = got[0].astype(np.float64)
    assert np.abs(g64.T @ g64 - np.eye(n)).max() <= (1e-12 if dtype == np.float64 else 2e-5)
