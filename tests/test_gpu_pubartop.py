"""pubarTop_pt's one block with 256 threads (up to 2048 columns) and with 1024,
against the C restatement. Its sums of NX terms carry at most NX 2^-53 of their
terms' magnitudes (1e-12); u, w and K as stored in FP32 are off by 2^-24 of
themselves each (1e-5).
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("NX", [31, 2048, 2080, 8192])
def test_pubartop_on_rows_of_any_length(NX, precision):
    from oracle.models import PortModel
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import random_state
    build.build()
    st = random_state(NX, 8, seed=NX)
    m = PortModel(st.grid)
    m.load(st)
    m.call("pubarTop_pt")
    ref = m.dump().scalars
    g = G.VVMGpu(st.grid, precision=precision)
    g.upload(st)
    g.call("pubartop")
    out = g.download().scalars
    g.close()
    assert ref["ubarTopp"] != ref["ubarTop"]
    tol = 1e-12 if precision == 0 else 1e-5
    assert abs(out["ubarTopp"] - ref["ubarTopp"]) <= tol * max(abs(ref["ubarTopp"]), 1.0)
