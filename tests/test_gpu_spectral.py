"""The Fourier-mode solver (VVM_SOLVER_SPECTRAL) against the reference and
against the multigrid-PCG path.

The Fourier-mode solve is the exact inverse of the cal_w operator up to
round-off: it is applied directly and its FP64 residual checked, so no CG
iteration normally follows (last_solve reports those iterations). The
reference comparisons use the same relative-L2 tolerances as the multigrid
path (tests/test_gpu_step.py).
"""
import numpy as np
import pytest

from conftest import golden, rel_l2
from tests_helpers import domain_means

PROG = ("zeta", "th", "qv", "qc", "qr", "u", "w")


@pytest.fixture(scope="module")
def gpu():
    from vvm_b200 import build, gpu as G
    build.build()
    return G


def test_spectral_rejects_non_power_of_two_nx():
    """Checked by create() before any device call (runs without a GPU)."""
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import GridSpec
    build.build()
    with pytest.raises(G.VVMGpuError) as e:
        G.VVMGpu(GridSpec(96, 32, 200.0, 200.0, 1.0), solver=G.VVM_SOLVER_SPECTRAL)
    assert e.value.code == 1 and "power of two" in str(e.value)


@pytest.mark.gpu
def test_spectral_poisson_manufactured_solution(gpu):
    from vvm_b200.initial_state import warm_bubble
    from oracle.models import PortModel
    z = golden("poisson_kat.npz")
    st = warm_bubble(int(z["NX"]), int(z["NZ"]))
    g = gpu.VVMGpu(st.grid, warm_start=False, solver=gpu.VVM_SOLVER_SPECTRAL)
    g.upload(st)
    W, it, rel = g.poisson_solve(z["b"], tol=1e-10)
    assert rel <= 1e-13 and it <= 1, (it, rel)   # CG iterations after the direct solve
    m = PortModel(st.grid)
    m.load(st)
    assert rel_l2(m.apply_A(W), z["b"]) <= 1e-13
    assert rel_l2(W, z["x_ans"]) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("nstep,tol_dyn,tol_th", [(1, 1e-9, 1e-13), (10, 1e-8, 1e-12)])
def test_spectral_fp64_steps_match_reference(gpu, nstep, tol_dyn, tol_th):
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble()
    g = gpu.VVMGpu(st.grid, solver=gpu.VVM_SOLVER_SPECTRAL)
    g.upload(st)
    g.step(nstep)
    out = g.download()
    z = golden(f"config1_step{nstep}.npz")
    for f in PROG:
        tol = tol_th if f in ("th", "qv") else tol_dyn
        assert rel_l2(out.fields[f], z[f]) <= tol, (f, rel_l2(out.fields[f], z[f]))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_spectral_graph_path_equals_host_loop_path(gpu, precision):
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble(128, 64)
    a = gpu.VVMGpu(st.grid, precision=precision, solver=gpu.VVM_SOLVER_SPECTRAL)
    a.upload(st)
    a.step(6)
    b = gpu.VVMGpu(st.grid, precision=precision, solver=gpu.VVM_SOLVER_SPECTRAL)
    b.upload(st)
    b.profile(True)
    b.step(6)
    da, db = a.download(), b.download()
    for f in PROG:
        assert np.array_equal(da.fields[f], db.fields[f]), f
    ia, ra = a.last_solve()
    ib, rb = b.last_solve()
    assert ia == ib and ra == rb and ra <= 1e-10


@pytest.mark.gpu
def test_spectral_and_multigrid_agree_at_2048x256(gpu):
    """Five steps of the benchmark grid with both solvers: the states agree
    to the solvers' tolerance."""
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble(2048, 256, 100.0, 100.0)
    out = {}
    for s in (gpu.VVM_SOLVER_MGPCG, gpu.VVM_SOLVER_SPECTRAL):
        g = gpu.VVMGpu(st.grid, solver=s)
        g.upload(st)
        g.step(5)
        out[s] = g.download()
        it, rel = g.last_solve()
        assert rel <= 1e-10
        g.close()
    for f in PROG:
        e = rel_l2(out[gpu.VVM_SOLVER_SPECTRAL].fields[f], out[gpu.VVM_SOLVER_MGPCG].fields[f])
        assert e <= 1e-8, (f, e)


@pytest.mark.gpu
def test_spectral_largest_nx(gpu):
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble(8192, 32, 100.0, 100.0)
    g = gpu.VVMGpu(st.grid, solver=gpu.VVM_SOLVER_SPECTRAL)
    g.upload(st)
    g.step(2)
    out = g.download()
    assert all(np.isfinite(out.fields[f]).all() for f in PROG)
    it, rel = g.last_solve()
    assert rel <= 1e-12 and it <= 2


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_spectral_600_steps_domain_means(gpu, precision):
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble()
    g = gpu.VVMGpu(st.grid, precision=precision, solver=gpu.VVM_SOLVER_SPECTRAL)
    g.upload(st)
    g.step(600)
    out = g.download()
    z = golden("config1_600.npz")
    got = domain_means(out)
    ref = z["means"][-1]
    if precision == 0:
        assert abs(got[0] - ref[0]) / abs(ref[0]) <= 1e-10
        for j in (1, 2, 3, 4):
            assert abs(got[j] - ref[j]) <= 1e-6 * max(abs(ref[j]), 1e-30), (j, got[j], ref[j])
    else:
        assert abs(got[0] - ref[0]) / abs(ref[0]) <= 1e-4
        assert abs(got[4] - ref[4]) / abs(ref[4]) <= 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,d", [(8, 6, 2000.0), (16, 5, 1800.0), (32, 8, 1500.0), (64, 19, 800.0), (4096, 11, 1000.0)])
def test_spectral_cal_w_at_edge_sizes(gpu, nx, nz, d):
    """The right-hand side formed in the row transform, w stored by the
    inverse and the check, at two to sixteen rows (a lone last row, one block
    of the check): captured steps equal the multigrid solver's, whose
    residuals are at 1e-12 (an error of 1e-9 in W at these heights, three
    steps), and equal the steps without a graph bit for bit."""
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble(nx, nz, d, d)

    def run(solver, profile=False):
        g = gpu.VVMGpu(st.grid, solver=solver, poisson_tol=1e-12)
        g.upload(st)
        if profile:
            g.profile(True)
        g.step(3)
        out, last = g.download(), g.last_solve()
        g.close()
        return out.fields, last

    a, la = run(gpu.VVM_SOLVER_SPECTRAL)
    b, lb = run(gpu.VVM_SOLVER_SPECTRAL, profile=True)
    m, _ = run(gpu.VVM_SOLVER_MGPCG)
    assert la == lb and la[1] <= 1e-12
    for f in PROG:
        assert np.array_equal(a[f], b[f]), f
    for f in ("w", "u"):
        assert np.abs(m[f]).max() > 0
        assert rel_l2(a[f], m[f]) <= 1e-8, (f, rel_l2(a[f], m[f]))


@pytest.mark.gpu
@pytest.mark.parametrize("nk", [3, 4, 16, 31, 33, 255, 256, 257])
def test_spectral_modes_at_every_height(gpu, nk):
    """The z solve in registers (to 256 rows) and beyond: the direct solve of a
    random right-hand side leaves a residual at round-off (1e-12: the
    operator's condition number at 257 rows of 32 columns, about 1e4, times
    2^-53 times the transforms' growth), without CG iterations."""
    from vvm_b200.initial_state import warm_bubble
    from oracle.models import PortModel
    nx, nz = 32, nk + 1
    st = warm_bubble(nx, nz, 200.0, 15000.0 / nz)
    g = gpu.VVMGpu(st.grid, warm_start=False, solver=gpu.VVM_SOLVER_SPECTRAL)
    g.upload(st)
    m = PortModel(st.grid)
    m.load(st)
    b = np.random.default_rng(nk).standard_normal(nx * nk)
    W, it, rel = g.poisson_solve(b, tol=1e-10)
    g.close()
    assert it == 0 and rel <= 1e-12
    assert rel_l2(m.apply_A(W), b) <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("tol,passes", [(1e-10, False), (1e-14, False), (1e-10, True), (1e-14, True)])
def test_captured_steps_do_their_end_over(gpu, tol, passes, precision):
    """Steps whose check fails (tol 1e-14), whose sweep needs the repeated passes
    or both: step graphs, whose end does over what the step went on with, equal
    the host's loops bit for bit, however the calls are cut, with moisture
    nudging after the diffusion and the counts of launches alike."""
    from vvm_b200.initial_state import warm_bubble
    if passes:
        st = warm_bubble(128, 24, 40.0, 40.0, 30.0 if precision else 10.0, amp=0.2, radius=400.0, zc=400.0)
    else:
        st = warm_bubble(128, 48)
    st.grid.moisture_nudge_time = 600.0
    runs, iters, launched = [], [], []
    for profile, calls in ((True, [11]), (False, [11]), (False, [1] * 11), (False, [3, 8])):
        g = gpu.VVMGpu(st.grid, precision=precision, solver=gpu.VVM_SOLVER_SPECTRAL, poisson_tol=tol)
        g.upload(st)
        if profile:
            g.profile(True)
        its = 0
        for n in calls:
            g.step(n)
            its += g.last_solve()[0]
        out = g.download()
        launched.append(g.launch_count)
        runs.append((out, g.last_solve()))
        iters.append(its)
        g.close()
    assert (iters[2] > 0) == (tol == 1e-14)
    for out, last in runs[1:]:
        assert last == runs[0][1]
        for f in PROG:
            assert np.isfinite(out.fields[f]).all() and np.array_equal(out.fields[f], runs[0][0].fields[f]), f
    assert launched[1] == launched[2] == launched[3]


@pytest.mark.gpu
def test_spectral_solve_edges(gpu):
    """What the check sees beside a passing solve: no right-hand side (W = 0,
    nothing to iterate), a NaN in it (refused as not converged) and, after
    those, an ordinary solve again."""
    from vvm_b200.initial_state import warm_bubble
    st = warm_bubble(64, 33)
    g = gpu.VVMGpu(st.grid, solver=gpu.VVM_SOLVER_SPECTRAL)
    g.upload(st)
    b = np.random.default_rng(3).standard_normal(64 * 32)
    first, it, rel = g.poisson_solve(b, tol=1e-10)
    assert it == 0 and 0 < rel <= 1e-12
    W, it, rel = g.poisson_solve(np.zeros_like(b), tol=1e-10)
    assert it == 0 and rel == 0 and not W.any()
    bad = b.copy()
    bad[7] = np.nan
    with pytest.raises(gpu.VVMGpuError) as e:
        g.poisson_solve(bad, tol=1e-10)
    assert "tolerance" in str(e.value)
    W, it, rel = g.poisson_solve(b, tol=1e-10)
    assert np.array_equal(W, first) and it == 0
    g.close()
