"""Assembly at the edges of its row and run classes, bit-exact against numpy:
rows around one warp's 32 / 64 pairs, the 256-pair limit of a warp, one
and several 4,096-pair tiles of the long-row sort; runs around the 64 sources
that one thread sums; the matrix read back to device and to host memory."""
import numpy as np
import pytest

from conftest import to_dev

pytestmark = pytest.mark.gpu


def _expected(nb, rows, cols, vals):
    keep = np.nonzero((rows >= 0) & (rows <= cols))[0]
    key = rows[keep].astype(np.int64) * nb + cols[keep]
    uniq, inv = np.unique(key, return_inverse=True)
    out = np.zeros((uniq.size, 9))
    np.add.at(out, inv, vals[keep])  # unbuffered: source order
    rowptr = np.zeros(nb + 1, np.int64)
    rowptr[1:] = np.cumsum(np.bincount(uniq // nb, minlength=nb))
    return rowptr, uniq % nb, out


@pytest.mark.parametrize("length", [1, 32, 33, 64, 65, 255, 256, 257, 1000, 4096, 4097, 8193, 20001])
@pytest.mark.parametrize("spread", [1, 7, 400])
def test_long_rows_and_runs(solver, cuda, length, spread):
    """One row of `length` pairs over `spread` columns (runs of length /
    spread sources), a second such row, and ordinary rows between."""
    import torch

    rng = np.random.default_rng(length * 1000 + spread)
    nb = 500
    r = [np.full(length, 3), np.full(length, 90), rng.integers(0, nb, 2000)]
    c = [3 + rng.integers(0, spread, length), 90 + rng.integers(0, spread, length), rng.integers(0, nb, 2000)]
    rows, cols = np.concatenate(r).astype(np.int32), np.concatenate(c).astype(np.int32)
    rows[-5:] = -1
    perm = rng.permutation(rows.size)
    rows, cols = rows[perm], cols[perm]
    vals = rng.normal(size=(rows.size, 9))
    solver.assemble(nb, to_dev(rows, cuda), to_dev(cols, cuda), to_dev(vals, cuda))
    rowptr, col, val = _expected(nb, rows, cols, vals)
    rp, ci, v = solver.upper_bsr()
    assert np.array_equal(rp, rowptr) and np.array_equal(ci, col) and np.array_equal(v, val)
    d = torch.empty(val.shape, dtype=torch.float64, device=cuda)
    solver._check(solver.lib.b2s_get_upper_bsr(solver.h, None, None, d.data_ptr()))
    assert np.array_equal(d.cpu().numpy(), val)


@pytest.mark.parametrize("nb", [1, 255, 256, 257, 1000])
def test_blocks_out_to_device_and_host(solver, cuda, nb):
    import torch

    rng = np.random.default_rng(nb)
    idx = np.arange(nb, dtype=np.int32)
    vals = rng.normal(size=(nb, 9))
    solver.assemble(nb, to_dev(idx, cuda), to_dev(idx, cuda), to_dev(vals, cuda))
    d = torch.full((nb + 1, 9), 7.0, dtype=torch.float64, device=cuda)
    solver._check(solver.lib.b2s_get_upper_bsr(solver.h, None, None, d.data_ptr()))
    assert np.array_equal(d[:nb].cpu().numpy(), vals) and (d[nb] == 7.0).all()
    assert np.array_equal(solver.upper_bsr()[2], vals)
