"""Left folds of long rows by a warp (vg_warp_fold) against the oracle's serial sums, bit for
bit, through both degree entry points (GPU): lengths around its steps and the serial limit,
and values that stop its integer prefix sums: doublings, exact ties, zeros, negative and
non-finite values, subnormals, sums outside the normal range."""
import numpy as np
import pytest

from oracle import vite_oracle as vo

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 64, 65, 255, 256, 257, 511, 512, 513, 767, 768, 1025, 5000, 40001]


def values(kind, n, rng):
    if kind == "u01":
        return rng.random(n)
    if kind == "wide":
        return np.exp(rng.uniform(-30.0, 30.0, n))
    if kind == "ties":  # eighths onto a large first value: every sum is a tie or nearly one
        x = rng.integers(0, 64, n) / 8.0
        if n:
            x[0] = 2.0**50
        return x
    if kind == "some_ties":
        x = rng.random(n)
        x[rng.random(n) < 0.01] = 2.0**-41
        return x
    if kind == "zeros":
        return np.where(rng.random(n) < 0.9, 0.0, rng.random(n))
    if kind == "signed":
        return rng.normal(size=n)
    if kind == "few_negative":
        x = rng.random(n)
        x[rng.random(n) < 0.002] *= -300.0
        return x
    if kind == "subnormal":
        return rng.integers(0, 50, n) * 5e-324
    if kind == "huge":
        return rng.random(n) * 1e306
    if kind == "inf":
        x = rng.random(n)
        if n > 600:
            x[600] = np.inf
        return x
    x = rng.random(n)
    if n > 300:
        x[300] = np.nan
    return x


@pytest.mark.parametrize("kind", ["u01", "wide", "ties", "some_ties", "zeros", "signed",
                                  "few_negative", "subnormal", "huge", "inf", "nan"])
def test_long_rows_fold_in_order(ctx, kind):
    import torch

    import vite_b200

    rng = np.random.default_rng(17)
    rows = [values(kind, n, rng) for n in LENGTHS + LENGTHS]
    rowptr = np.zeros(len(rows) + 1, np.int64)
    rowptr[1:] = np.cumsum([len(r) for r in rows])
    w = np.concatenate(rows)
    tail = rng.integers(0, len(rows), len(w))
    ref, _ = vo.vertex_degree(vo.Graph(rowptr, tail, w))
    got, _ = ctx.vertex_degree(ctx.upload(rowptr, tail, w))
    rp, wd = torch.from_numpy(rowptr).cuda(), torch.from_numpy(w).cuda()
    out = torch.empty(len(rows), dtype=torch.float64, device="cuda")
    vite_b200.vertex_degree_noalloc(len(rows), rp.data_ptr(), wd.data_ptr(), out.data_ptr())
    for x in (got, out.cpu().numpy()):
        np.testing.assert_array_equal(np.isnan(x), np.isnan(ref))
        ok = ~np.isnan(ref)
        np.testing.assert_array_equal(x[ok].view(np.int64), ref[ok].view(np.int64))
