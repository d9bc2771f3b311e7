"""The PCG in MAS slot order against direct solves: padded parts, vertices left
out of the partition, block rows outside the MAS range on both sides, an empty
row, affine bodies, x0 given or not, FP64 and mixed, graph and stream-ordered;
the same handle used again with another partition and another matrix size."""
import numpy as np
import pytest

from conftest import to_dev

pytestmark = pytest.mark.gpu


def _system(rng, n, before, after, bodies):
    """SPD block system: 4*bodies body rows, `before` rows, n mesh rows, `after`
    rows, the last of them empty; a random mesh graph with couplings out of it."""
    nb = 4 * bodies + before + n + after
    off = 4 * bodies + before
    edges = {(min(a, b), max(a, b)) for a in range(n) for b in (a + 1, a + 2, a + 5, a + 11) if b < n}
    rows, cols, vals = [], [], []

    def add(i, j, B):
        if i > j:
            i, j, B = j, i, B.T
        rows.append(i), cols.append(j), vals.append(B.T.ravel())

    last = nb - 1 if after else nb
    links = [(off + a, off + b) for a, b in sorted(edges)]
    links += [(int(rng.integers(0, off)), off + int(rng.integers(0, n))) for _ in range(n // 8 if off else 0)]
    links += [(off + int(rng.integers(0, n)), int(rng.integers(off + n, last))) for _ in range(n // 8 if last > off + n else 0)]
    for i, j in links:
        Q = rng.normal(size=(3, 3))
        K = Q @ Q.T + 0.1 * np.eye(3)
        add(i, i, K), add(j, j, K), add(i, j, -K)
    for i in range(last):
        add(i, i, 0.3 * np.eye(3))
    for b in range(bodies):
        Q = rng.normal(size=(12, 12))
        M = Q @ Q.T + np.eye(12)
        for i in range(4):
            for j in range(4):
                add(4 * b + i, 4 * b + j, M[3 * i:3 * i + 3, 3 * j:3 * j + 3]) if i <= j else None
    rows, cols, vals = np.array(rows, np.int32), np.array(cols, np.int32), np.array(vals)
    A = np.zeros((3 * nb, 3 * nb))
    for i, j, v in zip(rows, cols, vals):
        B = v.reshape(3, 3).T
        A[3 * i:3 * i + 3, 3 * j:3 * j + 3] += B
        if i != j:
            A[3 * j:3 * j + 3, 3 * i:3 * i + 3] += B.T
    e = np.array(sorted(edges) + [(b, a) for a, b in sorted(edges)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    start = np.zeros(n + 1, np.int32)
    start[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    return nb, off, rows, cols, vals, A, last, start, e[:, 1].astype(np.int32)


def _maps(rng, n, part, skip):
    """Parts of `part` consecutive vertices padded to 16, holes anywhere in a
    bank, `skip` vertices unpartitioned."""
    out = rng.permutation(n)[:skip]
    keep = np.setdiff1d(np.arange(n), out)
    p2r = []
    for k in range(0, keep.size, part):
        lanes = np.full(16, -1)
        vs = keep[k:k + part]
        lanes[np.sort(rng.permutation(16)[:vs.size])] = vs
        p2r.append(lanes)
    p2r = np.concatenate(p2r).astype(np.int32)
    r2p = np.full(n, -1, np.int32)
    r2p[p2r[p2r >= 0]] = np.nonzero(p2r >= 0)[0]
    return p2r, r2p


@pytest.mark.parametrize("n,before,after,bodies,part,skip", [
    (16, 0, 0, 0, 16, 0), (40, 0, 0, 0, 13, 0), (130, 5, 0, 0, 16, 7), (333, 0, 9, 0, 11, 0), (300, 3, 4, 3, 16, 40)])
@pytest.mark.parametrize("precision", [0, 1])
def test_pcg_in_slot_order(solver, cuda, n, before, after, bodies, part, skip, precision):
    import torch

    rng = np.random.default_rng(n + precision)
    for again in range(2):  # a second matrix and partition on the same handle
        nb, off, rows, cols, vals, A, last, start, lst = _system(rng, n - again, before, after, bodies)
        m = n - again
        solver.assemble(nb, to_dev(rows, cuda), to_dev(cols, cuda), to_dev(vals, cuda))
        solver.abd_init(0, 0)
        solver.mas_init(off, m, start, lst, *_maps(rng, m, part, skip))
        solver.abd_init(0, bodies)
        solver.precond_assemble(2)
        b = rng.normal(size=3 * nb)
        b[3 * last:] = 0.0
        ref = np.zeros(3 * nb)
        ref[:3 * last] = np.linalg.solve(A[:3 * last, :3 * last], b[:3 * last])
        bd = to_dev(b, cuda)
        for given, graph in ((False, True), (True, True), (True, False)):
            x = to_dev(ref + 0.1 * rng.normal(size=3 * nb) * (np.arange(3 * nb) < 3 * last), cuda)
            st = solver.pcg(bd, x, tol=1e-11, stop_rule=1, x0_given=given, precision=precision, use_graph=graph,
                            replace_every=10 if precision and graph else 0)
            assert st["converged"] == 1 and st["bypassed"] == 0
            # |dx| <= |A^-1| |r|, |r| <= 1e-11 |b|
            lim = 1e-11 * np.linalg.norm(b) * np.linalg.norm(np.linalg.inv(A[:3 * last, :3 * last]), 2) * 1.01
            assert np.linalg.norm(x.cpu().numpy() - ref) <= lim + 1e-13 * np.linalg.norm(ref)
        x = torch.full((3 * nb,), 7.0, dtype=torch.float64, device=cuda)
        st = solver.pcg(bd, x, tol=1e-11, stop_rule=1, precision=precision, max_iter=3)
        assert st["converged"] == 0 and bool(torch.isfinite(x).all())


@pytest.mark.parametrize("nb", [1, 300, 120000])
@pytest.mark.parametrize("precision", [0, 1])
def test_zero_right_hand_side_on_a_new_handle(solver, cuda, nb, precision):
    """b = 0 stops before the loop: the residual's sums run over more blocks
    than any sum before them on this handle."""
    import torch

    idx = torch.arange(nb, dtype=torch.int32, device=cuda)
    vals = torch.eye(3, dtype=torch.float64, device=cuda).reshape(1, 9).expand(nb, 9).contiguous()
    solver.assemble(nb, idx, idx, vals)
    solver.precond_assemble(1)
    x = torch.full((3 * nb,), 3.0, dtype=torch.float64, device=cuda)
    st = solver.pcg(torch.zeros_like(x), x, precision=precision)
    assert st["converged"] == 1 and st["rel_res"] == 0.0 and not x.any()


def _wide_system(rng, n, far=(1, 3, 41)):
    """n rows, couplings at the distances `far` (PSD per link) plus 0.3 I."""
    i = np.concatenate([np.arange(n - d) for d in far])
    j = i + np.repeat(far, [n - d for d in far])
    Q = rng.normal(size=(i.size, 3, 3))
    K = np.einsum("kab,kcb->kac", Q, Q)
    d = np.arange(n)
    rows = np.concatenate([i, j, i, d]).astype(np.int32)
    cols = np.concatenate([i, j, j, d]).astype(np.int32)
    vals = np.concatenate([K, K, -K, np.broadcast_to(0.3 * np.eye(3), (n, 3, 3))]).reshape(-1, 9)

    def product(x):
        x = x.reshape(n, 3)
        y, t = 0.3 * x, np.einsum("kab,kb->ka", K, x[i] - x[j])
        np.add.at(y, i, t)
        np.add.at(y, j, -t)
        return y.ravel()

    return rows, cols, vals, product


@pytest.mark.parametrize("n,part,edges,far", [
    (20003, 16, 0, (1, 3, 41)), (28001, 13, 2, (1, 3, 41)), (47003, 16, 4, (1, 3, 41)), (47900, 16, 4, (1, 3, 41)),
    (52007, 13, 0, (5,)), (56000, 16, 0, (5,)), (75773, 16, 2, (1,)), (75777, 16, 2, (1,))])
@pytest.mark.parametrize("precision", [0, 1])
def test_banks_of_many_components(solver, cuda, n, part, edges, far, precision):
    """A hierarchy whose banks fall into many components (mesh edges only inside
    runs of `edges` vertices), so every level has as many banks as blocks or
    more and a block takes several of a level in turn; sizes on either side of
    what the one-launch loop takes (3 or 5 blocks for each of 37,888 threads,
    75,776 rows)."""
    import torch

    rng = np.random.default_rng(n + precision)
    rows, cols, vals, product = _wide_system(rng, n, far)
    v = np.arange(n)
    e = v[(v + 1 < n) & ((v + 1) % max(edges, 1) != 0)] if edges else v[:0]
    e = np.concatenate([np.stack([e, e + 1], 1), np.stack([e + 1, e], 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    start = np.zeros(n + 1, np.int32)
    start[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    solver.assemble(n, to_dev(rows, cuda), to_dev(cols, cuda), to_dev(vals, cuda))
    solver.mas_init(0, n, start, e[:, 1].astype(np.int32), *_maps(rng, n, part, 0))
    solver.precond_assemble(2)
    b = rng.normal(size=3 * n)
    bd = to_dev(b, cuda)
    its = []
    for graph in (True, False):
        x = torch.zeros_like(bd)
        st = solver.pcg(bd, x, tol=1e-10, stop_rule=1, precision=precision, use_graph=graph, check_interval=1,
                        replace_every=50 if precision else 0)
        assert st["converged"] == 1 and st["bypassed"] == 0
        assert np.linalg.norm(b - product(x.cpu().numpy())) <= 1.01e-10 * np.linalg.norm(b)
        its.append(st["iterations_exact"])
    # the same recursion; the sums' order moves the stop by a few iterations,
    # and in FP32 the restarts from the true residual with it
    assert abs(its[0] - its[1]) <= (3 if precision == 0 else 0.2 * its[1])


@pytest.mark.parametrize("first", [56, 58, 72, 76])
@pytest.mark.parametrize("precision", [0, 1])
def test_body_rows_inside_the_mas_range(solver, cuda, first, precision):
    """An affine body whose rows a later b2s_mas_init covers, some of them in
    the partition and some not: rows of the partition take the MAS, the others
    the body's inverse with the residual of all four rows. The recursion in
    slot order follows the operator b2s_precond_apply shows, in one launch, in
    a graph and launch by launch."""
    import torch

    rng = np.random.default_rng(first)
    nb, off, rows, cols, vals, A, last, start, lst = _system(rng, 80, 0, 0, 0)
    p2r, r2p = _maps(rng, nb, 16, 0)
    out = np.arange(first + 1, first + 4, 2)  # two of the body's rows leave the partition
    p2r[r2p[out]] = -1
    r2p[out] = -1
    solver.assemble(nb, to_dev(rows, cuda), to_dev(cols, cuda), to_dev(vals, cuda))
    solver.abd_init(first, 1)
    solver.mas_init(0, nb, start, lst, p2r, r2p)
    solver.precond_assemble(2)
    n = 3 * nb
    z = torch.zeros(n, dtype=torch.float64 if precision == 0 else torch.float32, device=cuda)
    apply = solver.precond_apply if precision == 0 else solver.precond_apply_mixed
    P = np.zeros((n, n))
    for k in range(n):
        e = torch.zeros_like(z)
        e[k] = 1.0
        apply(e, z)
        P[:, k] = z.cpu().numpy()
    b = rng.normal(size=n)
    x, r = np.zeros(n), b.copy()
    p = s = P @ r
    rz0 = rz = r @ s
    for _ in range(4):
        a = rz / (p @ A @ p)
        x, r = x + a * p, r - a * (A @ p)
        s = P @ r
        p, rz = s + (r @ s) / rz * p, r @ s
    assert np.linalg.norm(P - P.T) > 1e-3 * np.linalg.norm(P)  # not the operator of any other reading of the range
    for graph, timing in ((True, False), (True, True), (False, False)):
        solver.set_timing(timing)
        xd = torch.zeros(n, dtype=torch.float64, device=cuda)
        st = solver.pcg(to_dev(b, cuda), xd, tol=1e-30, max_iter=5, precision=precision, use_graph=graph)
        # FP32 inverses and Z, or BF16 tiles with FP32 vectors whose residual
        # enters with 16 bits: 2^-24 and 2^-16 per apply, times the growth over four steps
        tol = 1e-5 if precision == 0 else 1e-2
        assert st["bypassed"] == 0 and abs(st["rz0"] - rz0) <= tol * rz0
        assert np.linalg.norm(xd.cpu().numpy() - x) <= tol * np.linalg.norm(x)


@pytest.mark.parametrize("precision", [0, 1])
def test_node_buffers_after_a_solve(solver, cuda, precision):
    """b2s_mas_get_nodes shows the last apply of the PCG whichever loop ran: every
    node's Z is its cluster's inverse times its R, and R_0 is the residual."""
    import torch

    rng = np.random.default_rng(5)
    n = 700
    rows, cols, vals, product = _wide_system(rng, n)
    start = np.zeros(n + 1, np.int32)
    v = np.arange(n - 1)
    e = np.concatenate([np.stack([v, v + 1], 1), np.stack([v + 1, v], 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    start[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    p2r, r2p = _maps(rng, n, 13, 0)
    solver.assemble(n, to_dev(rows, cuda), to_dev(cols, cuda), to_dev(vals, cuda))
    solver.mas_init(0, n, start, e[:, 1].astype(np.int32), p2r, r2p)
    solver.precond_assemble(2)
    b = rng.normal(size=3 * n)
    for graph in (True, False):
        for fresh in (0, 1):  # another solve: nothing of the first one may show
            bb = b if fresh else rng.normal(size=3 * n)
            x = torch.zeros(3 * n, dtype=torch.float64, device=cuda)
            solver.pcg(to_dev(bb, cuda), x, tol=1e-30, max_iter=4, check_interval=1, precision=precision, use_graph=graph)
        R, Z = solver.mas_nodes()
        r = np.zeros((p2r.size, 3))
        r[p2r >= 0] = (b - product(x.cpu().numpy())).reshape(n, 3)[p2r[p2r >= 0]]
        # the recursive residual: FP64, or FP32 over three updates
        assert np.abs(R[:p2r.size] - r).max() <= (1e-6 if precision == 0 else 1e-4) * np.abs(r).max()
        _, inv = solver.mas_clusters()
        M = np.zeros((len(inv), 16, 3, 16, 3))
        for k, (i, j) in enumerate((i, j) for i in range(16) for j in range(i, 16)):
            B = inv[:, k].reshape(-1, 3, 3).transpose(0, 2, 1)
            M[:, i, :, j] = B
            M[:, j, :, i] = B.transpose(0, 2, 1)
        M = M.reshape(len(inv), 48, 48).astype(np.float64)
        ref = np.einsum("cij,cj->ci", M, R.reshape(-1, 48).astype(np.float64))
        # FP32 products of 48 terms, or BF16 entries of the scaled inverse (2^-9 each)
        size = np.einsum("cij,cj->ci", np.abs(M), np.abs(R.reshape(-1, 48)).astype(np.float64))
        lim = 50 * 2.0**-24 * size if precision == 0 else 2.0**-8 * np.linalg.norm(size, axis=1, keepdims=True)
        assert (np.abs(Z.reshape(-1, 48) - ref) <= lim).all()
