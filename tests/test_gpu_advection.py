"""The scalar advection's tiles (31 columns by 8 rows a block, or by 32 where the
grid is large) at their edges: one step of a random state against the C
restatement. FP64 bars as for a step of the warm bubble (1e-12 for the advected
fields, 1e-9 for what the elliptic solve enters); the mixed step's fields
carry FP32 round-off (1e-5).
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("NX,NZ", [(4, 4), (30, 7), (31, 8), (32, 9), (62, 16), (64, 17), (1240, 121), (1248, 128)])
def test_step_matches_restatement(NX, NZ, precision):
    from oracle.models import PortModel
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import random_state
    build.build()
    st = random_state(NX, NZ, seed=NX + NZ)
    st.fields["qr"][st.fields["qr"] < 2e-4] = 0.0    # rain in part of the cells
    st.fields["qr"][0], st.fields["qr"][-1] = st.fields["qr"][-2], st.fields["qr"][1]
    m = PortModel(st.grid)
    m.load(st)
    m.one_step()
    ref = m.dump()
    g = G.VVMGpu(st.grid, precision=precision, poisson_tol=1e-12)
    g.upload(st)
    g.step(1)
    out = g.download()
    g.close()
    for n in ("th", "qv", "qc", "qr"):
        assert rel_l2(out.fields[n], ref.fields[n]) <= (1e-12 if precision == 0 else 1e-5), n
    for n in ("dth_advect", "dqv_advect", "dqc_advect", "dqr_advect", "dqr_VT"):
        assert rel_l2(out.hist[n], ref.hist[n]) <= (1e-12 if precision == 0 else 1e-4), n
    for n in ("zeta", "u", "w"):
        assert rel_l2(out.fields[n], ref.fields[n]) <= (1e-9 if precision == 0 else 1e-4), n
    assert rel_l2(out.precip, ref.precip) <= (1e-12 if precision == 0 else 1e-4)
