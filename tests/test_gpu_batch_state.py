"""What a batch does to its cases' state, in the orders a program may call it.

The autotuner straight after the upload, before any step: it builds the solver
on the way, and must leave it whole. Every case then steps as it does alone
with the tuned knobs, bit for bit, and a solve's residual, recomputed with the
C restatement's copy of the matrix, is what the solve reports: 1e-10 asked,
1e-9 allowed (the report is the same sum in another order, and a solve that
reports 1e-10 with a broken weight is off by all of its right-hand side).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PROG = ("zeta", "th", "qv", "qc", "qr", "u", "w")


@pytest.fixture(scope="module")
def G():
    from vvm_b200 import build, gpu
    build.build()
    return gpu


def _same(a, b):
    return all(np.array_equal(a.fields[f], b.fields[f]) for f in PROG)


@pytest.mark.parametrize("precision,solver,shapes", [
    (1, 2, [(64, 32), (64, 32), (128, 48)]),   # mixed, spectral, grouped and alone
    (0, 2, [(256, 32)]),
    (0, 0, [(64, 32), (96, 33)]),              # FP64, multigrid
    (1, 0, [(64, 32)]),
    (0, 1, [(64, 32)]),                        # the learned preconditioner, untrained
])
def test_autotune_before_the_first_step(G, port_lib, precision, solver, shapes):
    from vvm_b200.initial_state import warm_bubble
    sts = [warm_bubble(nx, nz, 200.0, 200.0, radius=max(400.0, nx * 25.0)) for nx, nz in shapes]
    b = G.VVMBatch([s.grid for s in sts], precision=precision, solver=solver)
    b.upload(sts)
    b.autotune(reps=1)
    b.step(4)
    b.synchronize()
    outs = [c.download() for c in b.cases]
    for c, st, out in zip(b.cases, sts, outs):
        g = G.VVMGpu(st.grid, precision=precision, solver=solver)
        g.set_tuning(*c.tuning())
        g.upload(st)
        g.step(4)
        assert _same(out, g.download())
        g.close()
        A = port_lib.PortModel(st.grid)
        A.load(st)
        rhs = np.random.default_rng(1).standard_normal(st.grid.NX * (st.grid.NZ - 1))
        W, _, rel = c.poisson_solve(rhs, tol=1e-10)
        assert rel <= 1e-10
        assert np.linalg.norm(rhs - A.apply_A(W)) <= 1e-9 * np.linalg.norm(rhs)
        A.close()
    b.close()


@pytest.mark.parametrize("NX", [4, 64, 1024, 2048, 8192])
def test_tuning_reports_the_row_fft_block_in_use(G, NX):
    """The automatic block is half a row, 32 to 1024 threads; setting what is
    reported changes nothing."""
    from vvm_b200.initial_state import warm_bubble
    g = G.VVMGpu(warm_bubble(NX, 8, 200.0, 200.0).grid, solver=G.VVM_SOLVER_SPECTRAL)
    auto = g.tuning()
    assert auto[1] == min(max(32, NX // 2), 1024)
    g.set_tuning(*auto)
    assert g.tuning() == auto
    g.set_tuning(0, 64)
    assert g.tuning()[1] == min(64, auto[1])
    g.close()


def test_autotune_keeps_the_tile_height(G):
    """The tile heights time alike (they shape passes a normal step does not
    run), so the autotuner tries none: it leaves the single pass as it is set
    or takes the cluster schedule. And it can come back from the cluster."""
    from vvm_b200.initial_state import warm_bubble
    sts = [warm_bubble(64, 32, 200.0, 200.0)] * 3
    for rows in (0, 32, 1, 1, 1):
        b = G.VVMBatch([s.grid for s in sts], precision=1, solver=G.VVM_SOLVER_SPECTRAL)
        for c in b.cases:
            c.set_tuning(rows, 0)
        b.upload(sts)
        b.step(3)
        b.autotune(reps=1)
        tr = {c.tuning()[0] for c in b.cases}
        assert len(tr) == 1 and tr <= {1, 32 if rows == 32 else 8}
        b.close()


@pytest.mark.parametrize("warm_start", [True, False])
@pytest.mark.parametrize("limit", [32, 0])   # grouped launches, cases as branches
def test_a_new_state_reaches_the_batch_graphs(G, warm_start, limit):
    """A second state with other profiles (density, and with it the elliptic
    operator and the diffusion's coefficients), uploaded after the batch has
    captured its steps: every case as alone, bit for bit. Then new knobs."""
    from vvm_b200.initial_state import warm_bubble
    old = [warm_bubble(64, 32, 200.0, 200.0, radius=800.0) for _ in range(3)]
    new = [warm_bubble(64, 32, 200.0, 200.0, radius=r, dthdz=6e-3, rh=0.5) for r in (600.0, 800.0, 1000.0)]
    b = G.VVMBatch([s.grid for s in old], precision=0, solver=G.VVM_SOLVER_SPECTRAL, warm_start=warm_start)
    b.grouping(limit)
    b.upload(old)
    b.step(6)
    b.upload(new)
    b.step(6)
    b.synchronize()
    outs = [c.download() for c in b.cases]
    for c in b.cases:
        c.set_tuning(1, 0)   # the cluster schedule: other last bits
    b.step(2)
    b.synchronize()
    for c, st, out in zip(b.cases, new, outs):
        g = G.VVMGpu(st.grid, precision=0, solver=G.VVM_SOLVER_SPECTRAL, warm_start=warm_start)
        g.upload(st)
        g.step(6)
        assert _same(out, g.download())
        g.set_tuning(1, 0)
        g.step(2)
        assert _same(c.download(), g.download())
        g.close()
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_a_member_that_holds_nan_is_stepped_like_any_other(G, precision):
    """A member of an ensemble has blown up: the first steps, driven by the
    host, take it as the captured ones do, and the others are as alone."""
    from vvm_b200.initial_state import warm_bubble
    sts = [warm_bubble(64, 32, 200.0, 200.0, amp=a, radius=800.0) for a in (1.0, 2.0, 3.0)]
    sts[1].fields["zeta"][20, 10] = np.nan
    b = G.VVMBatch([s.grid for s in sts], precision=precision, solver=G.VVM_SOLVER_SPECTRAL)
    b.upload(sts)
    for n in (1, 1, 1, 2):   # two steps by the host, three from graphs
        b.step(n)
    b.synchronize()
    outs = [c.download() for c in b.cases]
    assert np.isnan(outs[1].fields["w"]).any()
    b.close()
    for j in (0, 2):
        g = G.VVMGpu(sts[j].grid, precision=precision, solver=G.VVM_SOLVER_SPECTRAL)
        g.upload(sts[j])
        g.step(5)
        assert _same(outs[j], g.download())
        g.close()
    g = G.VVMGpu(sts[1].grid, precision=precision, solver=G.VVM_SOLVER_SPECTRAL)
    g.upload(sts[1])
    g.call("pzeta")
    g.call("cal_w")      # the routine takes it too
    assert np.isnan(g.download().fields["w"]).any()
    g.close()
