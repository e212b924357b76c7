"""The in-place diffusion sweep in one pass (and the repeated passes it asks for
when its coefficients are too large) against the sequential sweep of the C
restatement, at grids around its tiles: 108 owned columns (104 to 110 and 215
to 217 columns with ghosts), bands of 8 rows and one row more, the smallest
grid.

dt sets the size of the coefficients B + C ~ 2 K dt / dx^2 of the random state
(K up to ~100 m^2/s at dx = 200 m): a short tail (dt = 1), the long one (dt =
8), the repeated passes (dt = 60). Tolerance: a cell takes about 20 operations
on values of its neighbourhood, 20 * 2^-53 ~ 2e-15 relative in FP64 (bound
1e-13); the mixed step's K is itself formed in FP32 from differences of
neighbours (bound 1e-5).
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

PAIRS = (("zetap", 0), ("thp", 1), ("qvp", 2), ("qcp", 3), ("qrp", 4))


@pytest.fixture(scope="module")
def G():
    from vvm_b200 import build, gpu
    build.build()
    return gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dt", [1.0, 8.0, 60.0])
@pytest.mark.parametrize("NX,NZ", [(4, 4), (104, 8), (106, 9), (108, 17), (213, 16), (215, 25), (256, 40)])
def test_diffusion_matches_sequential_sweep(G, NX, NZ, dt, precision):
    from oracle.models import PortModel
    from vvm_b200.initial_state import random_state
    st = random_state(NX, NZ, dt=dt, seed=NX + NZ)
    rng = np.random.default_rng(NX)
    for n in ("zeta", "th", "qv", "qc", "qr"):
        st.fields[n + "p"] = st.fields[n] * (1.0 + 1e-3 * rng.standard_normal(st.fields[n].shape))
    m = PortModel(st.grid)
    m.load(st)
    m.call("RKM_RKH")
    ref = m.dump()
    g = G.VVMGpu(st.grid, precision=precision)
    g.upload(st)
    g.call("turbulence")
    out = g.download()
    g.close()
    for n, _ in PAIRS:
        assert rel_l2(out.fields[n], ref.fields[n]) <= (1e-13 if precision == 0 else 1e-5), n
    assert rel_l2(out.fields["qcp"], st.fields["qcp"]) > 1e-5   # it diffused


@pytest.mark.parametrize("precision,dt", [(0, 10.0), (1, 30.0)])
def test_repeated_passes_from_graphs(G, precision, dt):
    """Coefficients the single pass does not take (dx = 40 m, K = 10 m^2/s at
    least): the passes of a step graph and of a grouped launch give what the
    host's loop gives, bit for bit."""
    from vvm_b200.initial_state import warm_bubble
    sts = [warm_bubble(128, 24, 40.0, 40.0, dt, amp=a, radius=400.0, zc=400.0) for a in (0.1, 0.2)]
    host = []
    for st in sts:
        g = G.VVMGpu(st.grid, precision=precision, solver=G.VVM_SOLVER_SPECTRAL)
        g.upload(st)
        g.profile(True)      # timed steps run kernel by kernel from the host
        g.step(6)
        host.append(g.download())
        g.close()
        g = G.VVMGpu(st.grid, precision=precision, solver=G.VVM_SOLVER_SPECTRAL)
        g.upload(st)
        g.step(6)
        alone = g.download()
        g.close()
        for n in ("zeta", "th", "qv", "qc", "qr", "u", "w"):
            assert np.isfinite(alone.fields[n]).all() and np.array_equal(alone.fields[n], host[-1].fields[n]), n
    b = G.VVMBatch([st.grid for st in sts], precision=precision)
    b.upload(sts)
    b.step(6)
    b.synchronize()
    assert b.grouping() == 1
    for c, ref in zip(b.cases, host):
        out = c.download()
        for n in ("zeta", "th", "qv", "qc", "qr", "u", "w"):
            assert np.array_equal(out.fields[n], ref.fields[n]), n
    b.close()


def test_tails_over_a_whole_band_in_many_waves(G):
    """Tails of 8 rows and more (dx = 100 m, dt = 8 s: B + C = 2 K dt / dx^2 =
    0.016 at K's floor of 10 m^2/s, 9 rows) over bands of 8 rows, with more
    tiles in one launch than the GPU holds at once: 64 cases of 128 x 64, about
    2500 blocks. A band above the first starts at the ground then, and must
    leave the rows of the bands under it alone whichever of them ran before.
    Every case as alone, bit for bit (there all its tiles run at once)."""
    from vvm_b200.initial_state import warm_bubble
    kinds = [warm_bubble(128, 64, 100.0, 100.0, 8.0, amp=a, radius=800.0, zc=z) for a, z in ((0.2, 900.0), (0.4, 1200.0))]
    ref = []
    for st in kinds:
        g = G.VVMGpu(st.grid, solver=G.VVM_SOLVER_SPECTRAL)
        g.upload(st)
        g.step(5)
        ref.append(g.download())
        g.close()
        assert np.isfinite(ref[-1].fields["zeta"]).all()
    sts = [kinds[j % 2] for j in range(64)]
    b = G.VVMBatch([st.grid for st in sts], precision=0)
    b.grouping(64)
    b.upload(sts)
    b.step(5)
    b.synchronize()
    assert b.grouping() == 1
    for j, c in enumerate(b.cases):
        out = c.download()
        for n in ("zeta", "th", "qv", "qc", "qr", "u", "w", "RKM"):
            assert np.array_equal(out.fields[n], ref[j % 2].fields[n]), (j, n)
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_routine_turbulence_leaves_later_steps_alone(G, precision):
    """The largest eddy coefficient of a routine call (K at its cap of 8000
    m^2/s) does not reach the next captured step, which would ask for the
    repeated passes: the same kernels run and give the same bits as without
    the call."""
    from vvm_b200.initial_state import random_state, warm_bubble
    st = warm_bubble(128, 32, 200.0, 200.0, 4.0, radius=1000.0)
    wild = random_state(128, 32, dt=4.0, seed=3)
    for n in ("u", "w"):
        wild.fields[n] *= 40.0
    for n in ("zeta", "th", "qv", "qc", "qr"):
        wild.fields[n + "p"] = wild.fields[n]
    outs, counts = [], []
    for disturb in (False, True):
        g = G.VVMGpu(st.grid, precision=precision, solver=G.VVM_SOLVER_SPECTRAL, warm_start=False)
        g.upload(st)
        g.step(3)
        if disturb:
            g.upload(wild)
            g.call("turbulence")
            assert g.download().fields["RKM"].max() > 1000.0
            g.call("next_step")
        g.upload(st)
        n0 = g.launch_count
        g.step(2)
        counts.append(g.launch_count - n0)
        outs.append(g.download())
        g.close()
    assert counts[0] == counts[1]
    for n in ("zeta", "th", "qv", "qc", "qr", "u", "w", "RKM"):
        assert np.array_equal(outs[0].fields[n], outs[1].fields[n]), n


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("field,i,k", [("zeta", 5, 3), ("th", 107, 9), ("qc", 109, 24), ("qr", 200, 1)])
def test_a_value_that_is_not_finite_spreads_as_in_the_sequential_sweep(G, field, i, k, value, precision):
    """One such value reaches, through the recurrence, every cell above it and
    to its right, far past the tails by which the tiles find their inflows."""
    from oracle.models import PortModel
    from vvm_b200.initial_state import random_state
    st = random_state(215, 25, dt=1.0, seed=1)
    for n in ("zeta", "th", "qv", "qc", "qr"):
        st.fields[n + "p"] = st.fields[n].copy()
    st.fields[field + "p"][i, k] = value
    m = PortModel(st.grid)
    m.load(st)
    m.call("RKM_RKH")
    ref = m.dump()
    g = G.VVMGpu(st.grid, precision=precision)
    g.upload(st)
    g.call("turbulence")
    out = g.download()
    g.close()
    for n, _ in PAIRS:
        a, b = out.fields[n], ref.fields[n]
        ok = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), ok), n
        assert rel_l2(a[ok], b[ok]) <= (1e-13 if precision == 0 else 1e-5), n


@pytest.mark.parametrize("precision", [0, 1])
def test_steps_of_a_state_that_is_not_finite(G, precision):
    """The same in whole steps: captured ones (alone, and in a group beside
    sound cases) leave the bits of host-driven ones."""
    from vvm_b200.initial_state import warm_bubble
    st, bad = (warm_bubble(128, 40, 200.0, 200.0, radius=1000.0) for _ in range(2))
    bad.fields["th"][40, 12] = np.nan
    names = ("zeta", "th", "qv", "qc", "qr", "u", "w")
    # warm_start off: the second step on runs from a graph
    def alone(s, host):
        g = G.VVMGpu(s.grid, precision=precision, solver=G.VVM_SOLVER_SPECTRAL, warm_start=False)
        g.upload(s)
        if host:
            g.profile(True)
        for _ in range(3):
            g.step(1)
        out = g.download()
        g.close()
        return out
    ref = [alone(s, True) for s in (st, bad)]
    assert np.isfinite(ref[0].fields["zeta"]).all() and not np.isfinite(ref[1].fields["zeta"]).all()
    b = G.VVMBatch([s.grid for s in (st, bad, st)], precision=precision, warm_start=False)
    b.upload([st, bad, st])
    b.step(3)
    b.synchronize()
    assert b.grouping() == 1
    outs = [c.download() for c in b.cases]
    b.close()
    for out, r in ((alone(st, False), ref[0]), (alone(bad, False), ref[1]), (outs[0], ref[0]), (outs[1], ref[1]),
                   (outs[2], ref[0])):
        for n in names:
            assert np.array_equal(out.fields[n], r.fields[n], equal_nan=True), n
