"""Bounded waits of the elastic kernels, on chip and staged, at the batches that are
used: the wait-limit hook makes one run out without choosing other kernels, the
time-out is reported, and the next evaluation is right."""
import pytest

import hmclab_gb300 as H
import test_fwi_onchip as OC
from hmclab_gb300 import _lib
from hmclab_gb300.Helpers.CustomExceptions import DeviceTimeoutError
from test_fwi_strips import strips

pytestmark = pytest.mark.gpu
LIMIT_NS = 1_000_000


def test_the_hook_does_not_choose_the_kernels():
    """Forward and adjoint of a shot read one store: neither may depend on it."""
    for C in (1, 32, 64):
        (chip, _), _ = OC._pair(OC._config(60, 50, nt=4), C)
        before = strips(chip, C)
        with _lib.wait_limits(LIMIT_NS, withhold=True):
            assert min(before) > 0 and strips(chip, C) == before


@pytest.mark.parametrize("nx,C", [(60, 32), (60, 64), (256, 32)])
@pytest.mark.parametrize("call", ["misfit_batch", "gradient_batch"])
def test_a_wait_that_runs_out_is_reported(nx, C, call):
    (dist, direct), M = OC._pair(OC._config(nx, 40, nt=6), C)
    assert (strips(dist, C) == (0, 0)) == (nx == 256)
    want = getattr(direct, call)(M)
    hooked = H.Distributions.ElasticFullWaveform2D(dist)  # a copy captures its shots' graphs under the hook
    with _lib.wait_limits(LIMIT_NS, withhold=True):
        getattr(hooked, call)(M)
        want.cpu()
    with pytest.raises(DeviceTimeoutError):
        hooked.check_device_status()
    assert bool((getattr(dist, call)(M) == want).all())
    dist.check_device_status()
