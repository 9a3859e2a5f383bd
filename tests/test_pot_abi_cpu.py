"""Struct layout and host-side argument checks of the potential's fused
contractions and of the many-array Adam step (no GPU)."""
import ctypes

import pytest

from hmclab_gb300 import _lib
from tests.test_abi_cpu import lib, test_struct_layout_matches_c as layout  # noqa: F401


@pytest.mark.parametrize("cname, cls", [("hmc_pot_out", _lib.HmcPotOut), ("hmc_adam_array", _lib.HmcAdamArray)])
def test_layout(tmp_path, cname, cls):
    layout(tmp_path, cname, cls)


def test_rejected_on_the_host(lib):  # noqa: F811
    E, p = _lib.HMC_ERR_INVALID_ARG, 16
    o = _lib.HmcPotOut(z=p, ldz=4, out=p, ld_out=8, act=p, ld_act=8, act_t=p, ld_act_t=8, vec=p)

    def call(mode, N=4, **kw):
        for k, v in kw.items():
            setattr(o, k, v)
        return lib.hmc_tc_pot(mode, 4, N, 8, p, 8, p, 8, p, ctypes.byref(o), p, None)

    assert call(9) == E and b"unknown mode" in lib.hmc_last_error()
    assert call(_lib.HMC_POT_DELTA1, N=9) == E
    assert call(_lib.HMC_POT_DBAR1) == E and b"DBAR1" in lib.hmc_last_error()
    assert call(_lib.HMC_POT_ZBAR1) == E and b"aux" in lib.hmc_last_error()
    assert call(_lib.HMC_POT_DELTA2, act=None) == E
    assert call(_lib.HMC_POT_DBAR2, vec=None) == E
    a = (_lib.HmcAdamArray * 1)((3, p, p, p, None))
    assert lib.hmc_mlp_adam_many(1, a, 1e-3, 0.9, 0.999, 1e-8, 1, None) == E
    assert lib.hmc_mlp_adam_many(9, a, 1e-3, 0.9, 0.999, 1e-8, 1, None) == E
    assert lib.hmc_mlp_adam_many(1, a, 1e-3, 0.9, 0.999, 1e-8, 0, None) == E
