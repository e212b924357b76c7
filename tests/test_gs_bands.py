"""Which tile of the single-pass diffusion stores which row.

The tiles of one column chunk run in no order, so every row of a field must be
stored by exactly one band, and a band may store no row but those it owns and
the ghost row beside them: a row stored twice ends up with the value of
whichever tile came last. Counted here for every grid height, band height and
tail length of the kernel, from the rule the kernel itself compiles.
"""
import ctypes
import subprocess

import pytest

from conftest import REPO

CSRC = REPO / "2d-vector-vorticity-model_b200" / "csrc"

HARNESS = r"""
#include "gs_bands.cuh"
// stores[k]: how often a sweep stores row k, in the order k_gs_sweep does it:
// the ghost row under k0, the rows k0 .. kl, the ghost row over kl.
extern "C" int band_stores(int nz, int tr, int hz, int* stores) {
    const int nb = (nz - 2 + tr - 1) / tr;
    for (int b = 0; b < nb; b++) {
        const vvm::GSBand r = vvm::gs_band(b, tr, hz, nz);
        if (r.ks < 1 || r.ks > r.k0 || r.k0 > r.kl) return 1;
        if (r.bottom) stores[r.k0 - 1]++;
        for (int k = r.k0; k <= r.kl; k++) stores[k]++;
        if (r.top) stores[r.kl + 1]++;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("gs_bands")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-x", "c++", str(d / "h.cpp"), "-o", str(d / "h.so")],
                   check=True)
    return ctypes.CDLL(str(d / "h.so"))


@pytest.mark.parametrize("tr", [8, 16, 32])
def test_every_row_is_stored_once(lib, tr):
    for nz in range(6, 80):
        for hz in range(1, 17):
            stores = (ctypes.c_int * nz)()
            assert lib.band_stores(nz, tr, hz, stores) == 0
            assert list(stores) == [1] * nz, (nz, hz)


def test_the_kernel_uses_the_rule():
    """No store of k_gs_sweep decides about a ghost row by anything else."""
    text = (CSRC / "step_kernels.cuh").read_text()
    body = text[text.index(" gs_sweep_tile("):text.index(" k_gs_sweep_body(")]
    assert "gs_band(" in body and "band.bottom" in body and "band.top" in body
