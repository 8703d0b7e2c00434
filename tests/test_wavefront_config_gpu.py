"""A context that was given a configuration, or tuned, treats what the caller did
not ask for as an unconfigured one does: the same kernels are launched for a call
of few paths (the finish kernel alone, behind the first camera paths)."""
import ctypes as C

import numpy as np
import pytest

from walkray_gb300 import _lib as L
from walkray_gb300 import scenes as S
from walkray_gb300.api import Context

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def preview(built):
    """launches(configure): kernels of a 160x120 one-sample call after `configure(context, scene)`, and its image."""

    def call(configure):
        with Context() as c:
            sid = c.upload(S.cornell(160, 120))
            configure(c, sid)
            n = [C.c_uint64(), C.c_uint64()]
            c.lib.wr_kernel_launches(c.h, C.byref(n[0]))
            img = c.render(sid, 1, 8, seed=3, mode="wavefront")
            c.lib.wr_kernel_launches(c.h, C.byref(n[1]))
            return n[1].value - n[0].value, img

    return call


@pytest.mark.parametrize("how", ["capacity", "another knob", "by scene", "tuned"])
def test_few_paths_leave_the_loop(preview, how):
    configure = {"capacity": lambda c, s: c.set_wavefront_config(capacity=1 << 20),
                 "another knob": lambda c, s: c.set_wavefront_config(capacity=1 << 24, pixel_tile=8),
                 "by scene": lambda c, s: c.set_wavefront_config(capacity=1 << 24, drain_paths=-1),
                 "tuned": lambda c, s: c.autotune(s, 4, 8)}[how]
    want, image = preview(lambda c, s: None)
    got, configured = preview(configure)
    assert got == want
    assert np.allclose(configured, image, rtol=1e-4, atol=1e-5)


def test_the_range_of_drain_paths(preview):
    def refused(c, s):
        with pytest.raises(L.WRError):
            c.set_wavefront_config(capacity=1 << 24, drain_paths=-2)

    loop, _ = preview(lambda c, s: c.set_wavefront_config(capacity=1 << 24, drain_paths=0))
    finish, _ = preview(refused)
    assert loop > finish  # 0: never
