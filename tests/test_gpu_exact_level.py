"""The multigrid solver's exact last level at column counts where its row
transform can go wrong: below and around one tile (32 modes, 16 rows, 32
staged terms), odd counts, counts with an odd factor, and rows long enough
that levels are coarsened before it (4160 = 65 * 64).

Against the same system solved in numpy (FFT along x, one tridiagonal system
a mode). The solve stops at ||b - A W|| / ||b|| <= 1e-12; the operator's
smallest eigenvalue bounds what that residual leaves in W: for these grids
(levels at most NK rows, coefficients within a factor 3 of 1) at most about
NK^2 times the residual, so 1e-12 * 65^2 < 1e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve_numpy(b, up, dn):
    NK, NX = b.shape
    r = np.fft.rfft(b, axis=1)
    lam = -4.0 * np.sin(np.pi * np.arange(r.shape[1]) / NX) ** 2
    cp, x = np.zeros_like(r, dtype=float), np.zeros_like(r)
    for k in range(NK):
        den = lam - (up[k] + dn[k]) - (dn[k] * cp[k - 1] if k else 0.0)
        cp[k] = (up[k] if k < NK - 1 else 0.0) / den
        x[k] = (r[k] - (dn[k] * x[k - 1] if k else 0.0)) / den
    for k in range(NK - 2, -1, -1):
        x[k] -= cp[k] * x[k + 1]
    return np.fft.irfft(x, n=NX, axis=1)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("NX,NZ", [(4, 4), (5, 17), (31, 18), (33, 34), (62, 16), (64, 33), (222, 64), (255, 20),
                                   (500, 35), (1000, 18), (4096, 12), (4160, 14)])
def test_solve_matches_numpy(NX, NZ, precision):
    from vvm_b200 import build, gpu as G
    from vvm_b200.initial_state import warm_bubble
    build.build()
    st = warm_bubble(NX, NZ, 200.0, 200.0)
    b = np.random.default_rng(NX * 1000 + NZ).standard_normal((NZ - 1, NX))
    g = G.VVMGpu(st.grid, precision=precision, solver=G.VVM_SOLVER_MGPCG, warm_start=False)
    g.upload(st)
    W, it, rel = g.poisson_solve(b.reshape(-1), tol=1e-12)
    g.close()
    rhou, rhow, k = st.prof["rhou"], st.prof["rhow"], np.arange(2, NZ + 1)
    ref = _solve_numpy(b, rhow[k] / rhou[k], rhow[k] / rhou[k - 1])
    assert rel <= 1e-12
    assert np.linalg.norm(W - ref.reshape(-1)) <= 1e-8 * np.linalg.norm(ref)
