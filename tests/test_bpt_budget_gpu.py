"""The memory budget of the bidirectional renderer counts what is allocated: two
lists of 4 B per pair of lengths and sample."""
import numpy as np
import pytest

from walkray_gb300 import scenes as S
from walkray_gb300.api import Context
from walkray_gb300._lib import WRError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bidirectional", "vcm"])
def test_a_call_that_fits_the_budget_runs(ctx, mode):
    s = S.cornell(64, 64)
    records = 32
    need = 64 * 64 * (2 * records * 64 + 8 * records * (records + 1))  # records and lists; the rest is below 2 %
    sid = ctx.upload(s)
    want = ctx.render(sid, 1, records - 2, seed=3, mode=mode)
    ctx.release(sid)
    with Context(memory_budget=need * 110 // 100) as small:
        sid = small.upload(s)
        assert np.allclose(small.render(sid, 1, records - 2, seed=3, mode=mode), want, rtol=1e-4, atol=1e-5)
    with Context(memory_budget=need) as less:
        sid = less.upload(s)
        with pytest.raises(WRError):
            less.render(sid, 1, records - 2, seed=3, mode=mode)
