"""The MAS restriction: the residual of every coarse node against sums in numpy,
and the same bits from every apply, whatever the order of the blocks."""
import numpy as np
import pytest

from conftest import to_dev
from test_gpu_pcg_order import _maps

pytestmark = pytest.mark.gpu

# vertices, vertices per part, vertices per run of mesh edges (0: no edges, every
# vertex a component of its bank; None: one chain)
HIERARCHIES = [(16, 16, None), (255, 13, 4), (4096, 16, None), (5000, 11, 0), (70000, 16, 3), (70000, 16, None),
               (300000, 16, None)]


def _build(solver, cuda, rng, n, part, edges):
    import torch

    v = np.arange(n - 1)
    e = v if edges is None else (v[(v + 1) % edges != 0] if edges else v[:0])
    e = np.concatenate([np.stack([e, e + 1], 1), np.stack([e + 1, e], 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    start = np.zeros(n + 1, np.int32)
    start[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    idx = torch.arange(n, dtype=torch.int32, device=cuda)
    solver.assemble(n, idx, idx, torch.eye(3, dtype=torch.float64, device=cuda).reshape(1, 9).expand(n, 9).contiguous())
    solver.mas_init(0, n, start, e[:, 1].astype(np.int32), *_maps(rng, n, part, 0))
    solver.precond_assemble(2)


@pytest.mark.parametrize("n,part,edges", HIERARCHIES)
@pytest.mark.parametrize("precision", [0, 1])
def test_restricted_residuals(solver, cuda, n, part, edges, precision):
    import torch

    rng = np.random.default_rng(n)
    _build(solver, cuda, rng, n, part, edges)
    begin, count, table = solver.mas_hierarchy(n)
    dt = torch.float64 if precision == 0 else torch.float32
    apply = solver.precond_apply if precision == 0 else solver.precond_apply_mixed
    r = rng.normal(size=(n, 3)).astype(np.float32)
    z = torch.zeros(3 * n, dtype=dt, device=cuda)
    for _ in range(2):  # the second apply finds the first one's entries
        apply(to_dev(r.ravel(), cuda, dt), z)
    R, _ = solver.mas_nodes()
    for l in range(1, len(begin) - 1):
        ref, size = np.zeros((len(R), 3)), np.zeros((len(R), 3))
        np.add.at(ref, table[:, l - 1], r.astype(np.float64))
        np.add.at(size, table[:, l - 1], np.abs(r))
        a, b = begin[l], begin[l] + count[l]
        # level 1 in FP32 over at most 16 lanes, the levels above FP64 sums of
        # those, rounded once
        assert (np.abs(R[a:b] - ref[a:b]) <= 17 * 2.0**-24 * size[a:b]).all()


@pytest.mark.parametrize("n,part,edges", HIERARCHIES[2:])
@pytest.mark.parametrize("precision", [0, 1])
def test_applies_are_reproducible(solver, cuda, n, part, edges, precision):
    """Residuals of +-2^40 among ones of order 1: another order of the FP64 sums
    is off by 2^-12 of them, far above the FP32 the sums are rounded to."""
    import torch

    rng = np.random.default_rng(n)
    _build(solver, cuda, rng, n, part, edges)
    r = rng.normal(size=(n, 3))
    big = rng.permutation(n)[:n // 32 * 2]
    r[big[::2]], r[big[1::2]] = 2.0**40, -(2.0**40)
    dt = torch.float64 if precision == 0 else torch.float32
    rd = to_dev(r.ravel(), cuda, dt)
    apply = solver.precond_apply if precision == 0 else solver.precond_apply_mixed
    first = None
    for _ in range(25):
        z = torch.zeros_like(rd)
        apply(rd, z)
        now = (z.cpu().numpy(), *solver.mas_nodes())
        first = first or now
        assert all(np.array_equal(a, b) for a, b in zip(first, now))
