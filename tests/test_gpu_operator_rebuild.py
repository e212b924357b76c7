"""A context that gets states of other density profiles builds its elliptic
operator anew in the memory of the one before: the device's free memory stays
where it was after both operators have been built once, and the steps are those
of a context that never saw the other state, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,precision,NX", [(0, 0, 2048), (0, 1, 1000), (2, 0, 2048), (1, 0, 512), (0, 0, 64),
                                                 (2, 1, 64)])
def test_new_densities_take_no_memory(solver, precision, NX):
    import torch
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import warm_bubble
    build.build()
    sts = [warm_bubble(NX, 64, 200.0, 200.0, dthdz=a) for a in (3e-3, 6e-3)]
    assert not np.array_equal(sts[0].prof["rhou"], sts[1].prof["rhou"])
    g = G.VVMGpu(sts[0].grid, precision=precision, solver=solver)
    free = []
    for j in range(8):
        g.upload(sts[j % 2])
        g.step(1)
        g.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    out = g.download()
    g.close()
    assert free[2:] == [free[1]] * 6
    if solver != 1:   # (the untrained network keeps the scales of the operator it was built with)
        g = G.VVMGpu(sts[1].grid, precision=precision, solver=solver)
        g.upload(sts[1])
        g.step(1)
        alone = g.download()
        g.close()
        for n in ("zeta", "th", "qv", "u", "w"):
            assert np.array_equal(out.fields[n], alone.fields[n]), n
