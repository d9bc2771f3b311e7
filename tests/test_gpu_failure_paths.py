"""The PCG's failure arms, driven by host-made inputs (no GPU fault involved).

* PSD guard (LinearFusedPCG::fused_pcg, linear_fused_pcg.cu:1843-1877): when
  r0.z0 < 0 or is not finite the preconditioner is bypassed and plain CG runs.
  A negated SPD system (A' = -A, b' = -b: the same solution) makes every
  block-Jacobi action negative definite, so r0.z0 < 0.
* Non-finite input (linear_fused_pcg.cu:1013-1060): a NaN in b is refused
  with B2S_ERR_NUMERIC before any iteration.
* Iteration cap (LinearPCG::pcg, linear_pcg.cu:420-435): with max_iter = 3 the
  solve stops unconverged and reports it.
* Warm start refused by its FP64 check: x0 = 0 (the plain start).
* A device wait that runs out (b2s_inject_failure shortens it): the call ends
  with B2S_ERR_CUDA and the handle solves again.
"""
import numpy as np
import pytest

from conftest import to_dev
from libuipc_b200 import _abi
from libuipc_b200.linear_system import B200SolveError, partition_maps, partition_rcb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

PRECISIONS = [_abi.B2S_PRECISION_FP64, _abi.B2S_PRECISION_MIXED]


def _setup(solver, s, dev, kind, negate=False):
    sign = -1.0 if negate else 1.0
    solver.assemble(s.n_verts, to_dev(s.rows, dev), to_dev(s.cols, dev), to_dev(sign * s.vals, dev))
    if kind == _abi.B2S_PRECOND_MAS:
        p2r, r2p = partition_maps(partition_rcb(s.positions))
        solver.mas_init(0, s.n_verts, s.adj_start, s.adj_list, p2r, r2p)
    solver.precond_assemble(kind)
    return to_dev(sign * s.b, dev)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_psd_guard_bypasses_an_indefinite_preconditioner(solver, cuda, cube5, precision):
    import torch

    b = _setup(solver, cube5, cuda, _abi.B2S_PRECOND_JACOBI, negate=True)
    x = torch.zeros_like(b)
    st = solver.pcg(b, x, tol=1e-6, stop_rule=_abi.B2S_STOP_RELRES, check_interval=1, precision=precision,
                    replace_every=50)
    assert st["bypassed"] == 1
    assert st["rz0"] > 0.0  # the plain start's r.r
    assert st["converged"] == 1 and st["rel_res"] <= 1e-6
    # the same arm in the oracle: bypassed too, and plain CG's iteration count
    A = O.OracleMatrix(cube5.n_verts, cube5.rows, cube5.cols, -cube5.vals)
    xo, info = O.pcg(A, -cube5.b, precond=O.ORC_PRECOND_JACOBI, tol=1e-6, stop_rule=O.ORC_STOP_RELRES)
    assert info["bypassed"] == 1 and info["converged"] == 1
    if precision == _abi.B2S_PRECISION_FP64:
        # plain CG over ~240 iterations: rounding (atomics in the SpMV) moves
        # the stop by a few iterations
        assert abs(st["iterations_exact"] - info["iterations"]) <= max(2, 0.05 * info["iterations"])
    # and, solved tightly, the solution is the unnegated system's
    x = torch.zeros_like(b)
    st = solver.pcg(b, x, tol=1e-11, stop_rule=_abi.B2S_STOP_RELRES, check_interval=5, precision=precision,
                    replace_every=50)
    assert st["bypassed"] == 1 and st["converged"] == 1
    A0 = O.OracleMatrix(cube5.n_verts, cube5.rows, cube5.cols, cube5.vals)
    xt, _, _ = O.cg_truth(A0, cube5.b, tol=1e-13)
    assert np.linalg.norm(x.cpu().numpy() - xt) <= 1e-6 * np.linalg.norm(xt)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_positive_definite_system_is_not_bypassed(solver, cuda, cube5, precision):
    import torch

    b = _setup(solver, cube5, cuda, _abi.B2S_PRECOND_MAS)
    x = torch.zeros_like(b)
    st = solver.pcg(b, x, tol=1e-4, stop_rule=_abi.B2S_STOP_RELRES, precision=precision)
    assert st["bypassed"] == 0 and st["converged"] == 1


@pytest.mark.parametrize("precision", PRECISIONS)
def test_nan_in_rhs_is_a_numeric_error(solver, cuda, cube5, precision):
    import torch

    b = _setup(solver, cube5, cuda, _abi.B2S_PRECOND_MAS)
    b[7] = float("nan")
    x = torch.zeros_like(b)
    with pytest.raises(B200SolveError) as ei:
        solver.pcg(b, x, tol=1e-4, stop_rule=_abi.B2S_STOP_RELRES, precision=precision)
    assert ei.value.code == _abi.B2S_ERR_NUMERIC
    # the handle stays usable: the next solve of a finite system works
    b[7] = 0.0
    st = solver.pcg(b, x, tol=1e-4, stop_rule=_abi.B2S_STOP_RELRES, precision=precision)
    assert st["converged"] == 1


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("use_graph", [True, False])
def test_iteration_cap_reports_not_converged(solver, cuda, cube5, precision, use_graph):
    import torch

    b = _setup(solver, cube5, cuda, _abi.B2S_PRECOND_JACOBI)
    x = torch.zeros_like(b)
    st = solver.pcg(b, x, tol=1e-10, stop_rule=_abi.B2S_STOP_RELRES, check_interval=1, max_iter=3,
                    precision=precision, use_graph=use_graph)
    assert st["converged"] == 0
    assert st["iterations"] == 3
    assert st["rel_res"] > 1e-10
    # x holds the third iterate (finite), and the solve can be resumed from it
    assert np.isfinite(x.cpu().numpy()).all() and np.isfinite(st["rel_res"])
    st2 = solver.pcg(b, x, tol=1e-6, stop_rule=_abi.B2S_STOP_RELRES, precision=precision, x0_given=True,
                     replace_every=50)
    assert st2["converged"] == 1 and st2["rel_res"] <= 1e-6


def test_warm_start_refused_by_its_check_is_zero(solver, cuda, cube5):
    """A start the FP64 check refuses falls back to x0 = 0: a history vector
    with a non-finite entry (its Galerkin coefficients are not finite), and
    random history vectors, which are kept only when the check passes."""
    import torch

    b = _setup(solver, cube5, cuda, _abi.B2S_PRECOND_MAS)
    solver.ws_init(hidden=64, seed=1)
    rng = np.random.default_rng(4)
    bad = to_dev(rng.standard_normal(3 * cube5.n_verts), cuda)
    bad[11] = float("inf")
    x0 = torch.full_like(b, 7.0)
    info = solver.ws_predict(b, x0, history=[bad], mode=_abi.B2S_WS_MODE_PREV)
    assert info["mode"] == _abi.B2S_WS_MODE_ZERO
    assert float(x0.abs().max()) == 0.0
    # random directions: either kept with a passing check, or zero
    junk = [to_dev(rng.standard_normal(3 * cube5.n_verts), cuda) for _ in range(3)]
    x1 = torch.full_like(b, 7.0)
    info = solver.ws_predict(b, x1, history=junk, mode=_abi.B2S_WS_MODE_HISTORY)
    if info["mode"] == _abi.B2S_WS_MODE_ZERO:
        assert float(x1.abs().max()) == 0.0
    else:
        assert info["rz_ratio"] < 1.0
    # and the PCG from the refused start is the plain solve
    st = solver.pcg(b, x0, tol=1e-4, stop_rule=_abi.B2S_STOP_RELRES, x0_given=True)
    xz = torch.zeros_like(b)
    st0 = solver.pcg(b, xz, tol=1e-4, stop_rule=_abi.B2S_STOP_RELRES)
    assert st["iterations_exact"] == st0["iterations_exact"]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("kind", [_abi.B2S_PRECOND_JACOBI, _abi.B2S_PRECOND_MAS])
@pytest.mark.parametrize("polls", [0, 1])
def test_a_barrier_that_runs_out_ends_the_call(solver, cuda, cube10, kind, precision, polls):
    """The one-launch PCG (1,331 rows) with barriers that give up after `polls`
    polls: the call returns an error, and the same handle, with the same build
    and with the default limit again, solves as it did before."""
    import torch

    b = _setup(solver, cube10, cuda, kind)
    args = dict(tol=1e-8, stop_rule=_abi.B2S_STOP_RELRES, precision=precision, replace_every=50)
    x0 = torch.zeros_like(b)
    st0 = solver.pcg(b, x0, **args)
    assert st0["converged"] == 1
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_WAIT_POLLS, polls))
    for _ in range(2):
        with pytest.raises(B200SolveError) as e:
            solver.pcg(b, torch.zeros_like(b), **args)
        assert e.value.code == _abi.B2S_ERR_CUDA and "timed out" in str(e.value)
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_WAIT_POLLS, -1))
    x = torch.zeros_like(b)
    st = solver.pcg(b, x, **args)
    # the two solves differ in the order of the SpMV's reductions only: the stop
    # may move by a few iterations, the answers by the tolerance's own error
    # (3e-7 of the solution on a cube at this tolerance)
    assert st["converged"] == 1 and abs(st["iterations_exact"] - st0["iterations_exact"]) <= 5
    assert float((x - x0).norm()) <= 1e-5 * float(x0.norm())


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("kind", [_abi.B2S_PRECOND_JACOBI, _abi.B2S_PRECOND_MAS])
@pytest.mark.parametrize("replace_every", [0, 20])
def test_a_refused_cooperative_launch_takes_the_steps(solver, cuda, cube10, kind, precision, replace_every):
    """Where the device refuses the one-launch PCG's grid, the same call runs
    launch by launch (the captured graph, in slot order with the MAS)."""
    import torch

    b = _setup(solver, cube10, cuda, kind)
    args = dict(tol=1e-8, stop_rule=_abi.B2S_STOP_RELRES, precision=precision, replace_every=replace_every)
    x0, x1 = torch.zeros_like(b), torch.zeros_like(b)
    solver.reset_timers()
    st0 = solver.pcg(b, x0, **args)
    one = solver.timers()["kernel_launches"]
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_LAUNCH, 1000))
    solver.reset_timers()
    st1 = solver.pcg(b, x1, **args)
    steps = solver.timers()["kernel_launches"]
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_LAUNCH, 0))
    assert st0["converged"] == st1["converged"] == 1
    assert steps >= 4 * st1["iterations_exact"] > one  # it did take the steps
    # as for the barriers above: rounding order only
    assert abs(st0["iterations_exact"] - st1["iterations_exact"]) <= 5
    assert float((x0 - x1).norm()) <= 1e-5 * float(x0.norm())


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("timing", [False, True])
def test_no_room_for_the_slot_order(cuda, cube5, precision, timing):
    """The MAS solve wants a copy of the matrix in slot order and vectors of that
    length. Whichever of its allocations fails, the call gives them back and
    solves in the matrix's own order; the next one has its copy again. timing:
    launch by launch, with the FP64 SpMV's tile ranks."""
    import torch

    from libuipc_b200.linear_system import Solver

    x0 = None
    for k in range(0, 22):  # 0: none fails; the last ones lie past the solve's allocations
        s = Solver(0)
        try:
            b = _setup(s, cube5, cuda, _abi.B2S_PRECOND_MAS)
            s.set_timing(timing)
            args = dict(tol=1e-8, stop_rule=_abi.B2S_STOP_RELRES, precision=precision, replace_every=50)
            s._check(s.lib.b2s_inject_failure(s.h, _abi.B2S_INJECT_ALLOC, k))
            x = torch.zeros_like(b)
            st = s.pcg(b, x, **args)
            s._check(s.lib.b2s_inject_failure(s.h, _abi.B2S_INJECT_ALLOC, 0))
            assert st["converged"] == 1 and st["rel_res"] <= 1e-8
            x0 = x if x0 is None else x0
            again = torch.zeros_like(b)
            assert s.pcg(b, again, **args)["converged"] == 1
            for v in (x, again):  # both stop at 1e-8: as for the barriers above
                assert float((v - x0).norm()) <= 1e-5 * float(x0.norm())
        finally:
            s.close()


def test_an_allocation_that_fails_is_a_cuda_error(solver, cuda, cube5):
    for k in (1, 2, 5):
        solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_ALLOC, k))
        with pytest.raises(B200SolveError) as e:
            _setup(solver, cube5, cuda, _abi.B2S_PRECOND_JACOBI)
        assert e.value.code == _abi.B2S_ERR_CUDA and "out of memory" in str(e.value)
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_ALLOC, 0))
    _setup(solver, cube5, cuda, _abi.B2S_PRECOND_JACOBI)


def test_products_after_the_first_allocate_nothing(solver, cuda, cube10):
    """The FP64 product builds its tile ranks from the second call of an assembly
    on, in room the assembly has made."""
    import torch

    b = _setup(solver, cube10, cuda, _abi.B2S_PRECOND_JACOBI)
    y = [torch.zeros_like(b) for _ in range(3)]
    solver.spmv(b, y[0])
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_ALLOC, 1))
    solver.spmv(b, y[1], with_dot=True)
    solver.spmv(b, y[2])
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_ALLOC, 0))
    for v in y[1:]:  # reductions in another order: a few ulp of the row sums
        assert float((v - y[0]).abs().max()) <= 1e-13 * float(y[0].abs().max())


@pytest.mark.parametrize("n_triplets", [1, 12, 10000, 10241, 60001])
def test_read_back_allocates_nothing(solver, cuda, n_triplets):
    """The blocks to host memory, in pieces through the assembly's scratch (5,120
    blocks while there are fewer than 36,864 triplets, then a ninth of 1.25 times
    those)."""
    rng = np.random.default_rng(n_triplets)
    idx = np.arange(n_triplets, dtype=np.int32) // 2  # two triplets per block
    vals = rng.normal(size=(n_triplets, 9))
    solver.assemble(n_triplets, to_dev(idx, cuda), to_dev(idx, cuda), to_dev(vals, cuda))
    ref = vals[0::2].copy()
    ref[:n_triplets // 2] += vals[1::2]
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_ALLOC, 1))
    _, col, v = solver.upper_bsr()
    solver._check(solver.lib.b2s_inject_failure(solver.h, _abi.B2S_INJECT_ALLOC, 0))
    assert np.array_equal(col, np.unique(idx)) and np.array_equal(v, ref)
