"""The binding's transfer of the prognostic fields, without a GPU: which
addresses reach the library."""
import ctypes

import numpy as np


class _Library:
    """Takes the calls of the binding and keeps the state they were given."""

    def vvm_gpu_download_prognostic(self, handle, ref):
        self.state = {n: ctypes.cast(getattr(ref._obj, n), ctypes.c_void_p).value
                      for n in ("zeta", "th", "qv", "qc", "qr", "u", "w", "RKM", "precip")}
        return 0


def test_download_prognostic_skips_fields_given_as_none():
    from vvm_b200 import gpu
    from vvm_b200.initial_state import warm_bubble
    lib = _Library()
    g = gpu.VVMGpu._borrow(lib, 1, warm_bubble(8, 8).grid, None)
    out = {n: np.zeros((10, 10)) for n in ("zeta", "th", "qv", "qc", "qr", "u", "w")}
    out["qc"] = out["w"] = None
    g.download_prognostic(out)
    for n in ("zeta", "th", "qv", "qr", "u"):
        assert lib.state[n] == out[n].ctypes.data
    assert lib.state["qc"] is None and lib.state["w"] is None
    assert lib.state["RKM"] is None and lib.state["precip"] is None
