"""RKM_RKH's branches where theta is not what it is in the atmosphere: zero,
negative, infinite, and differences so small that Ri rounds to zero. The
reference's test is on Ri alone (0 < Ri < 1/4 and Ri < 0, RKM_RKH in
Turbulent.cpp:5-45); the coefficients against the C restatement, FP64 to
round-off (a dozen operations, two roots: 1e-14, bound 1e-13).
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NX,NZ", [(64, 20), (2048, 80)])   # one row a thread, four
@pytest.mark.parametrize("kind", ["negative", "zero", "infinite", "mixed signs", "no stratification", "denormal"])
def test_eddy_coefficients_of_any_theta(kind, NX, NZ):
    from oracle.models import PortModel
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import random_state
    build.build()
    st = random_state(NX, NZ, seed=5)
    rng = np.random.default_rng(2)
    th = st.fields["th"].copy()
    if kind == "negative":
        th = -th
    elif kind == "zero":
        th[rng.random(th.shape) < 0.3] = 0.0
    elif kind == "infinite":
        th[20, 7] = np.inf
        th[40, 11] = -np.inf
    elif kind == "mixed signs":
        th *= np.where(rng.random(th.shape) < 0.5, 1.0, -1.0)
    elif kind == "no stratification":
        th[:] = 300.0
    else:   # differences whose Ri is below the smallest number
        th = np.where(rng.random(th.shape) < 0.5, 5e-324, 1e-323) + 0.0
    st.fields["thp"] = th
    for n in ("zeta", "qv", "qc", "qr"):
        st.fields[n + "p"] = st.fields[n].copy()
    m = PortModel(st.grid)
    m.load(st)
    with np.errstate(all="ignore"):
        m.call("RKM_RKH")
    ref = m.dump()
    g = G.VVMGpu(st.grid)
    g.upload(st)
    g.call("turbulence")
    out = g.download()
    g.close()
    for n in ("RKM", "RKH"):
        a, b = out.fields[n][1:-1, 1:-1], ref.fields[n][1:-1, 1:-1]
        assert np.array_equal(np.isnan(a), np.isnan(b)), n
        ok = ~np.isnan(b)
        assert np.abs(a[ok] - b[ok]).max() <= 1e-13 * np.abs(b[ok]).max(), n
        assert rel_l2(a[ok], b[ok]) <= 1e-13, n
