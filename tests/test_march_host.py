"""Host-side parts of the steps, without a GPU: what a step returns for its error bits."""
from __future__ import annotations

import ctypes

from conftest import load_pkg

hb = load_pkg()


def test_result_of_a_step_by_its_error_bits():
    """A step that reports a wait that gave up (bit 1) returns HYDRO_ERR_TIMEOUT, also where the
    state is non-physical (bit 0) too, and leaves its scratch words to be zeroed. The synchronous 2D
    and 3D steps and hydro_last_step_info share this mapping."""
    fn = hb.lib()["_ZN5hydro11step_resultEjPKcPb"]
    fn.argtypes = [ctypes.c_uint, ctypes.c_char_p, ctypes.POINTER(ctypes.c_bool)]
    for bits, rc, word in ((0, hb.HYDRO_OK, None), (1, hb.HYDRO_ERR_NONPHYSICAL, "non-physical"),
                           (2, hb.HYDRO_ERR_TIMEOUT, "timed out"), (3, hb.HYDRO_ERR_TIMEOUT, "timed out")):
        hb.lib().hydro_clear_error()
        dirty = ctypes.c_bool(False)
        assert fn(bits, b"step3d", ctypes.byref(dirty)) == rc
        assert dirty.value == (rc == hb.HYDRO_ERR_TIMEOUT)
        code, msg = hb.last_error()
        assert (code, bool(word) and word in msg and "step3d" in msg) == (rc, bool(word))
        assert fn(bits, None, ctypes.byref(dirty)) == rc
