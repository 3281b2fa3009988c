"""Ensembles of dry members, which have no moisture buffers: every member
equals its standalone context bit for bit, on basic states of height only and
on one that varies horizontally, with level counts of and off whole quads."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tune", [False, True])
@pytest.mark.parametrize("base", ["height", "varying"])
@pytest.mark.parametrize("nz", [16, 13])
@pytest.mark.parametrize("precision", [abi.GA_PREC_F64, abi.GA_PREC_F32], ids=["f64", "f32"])
def test_dry_members_equal_standalone_runs(precision, nz, base, tune):
    make = configs.dry_bubble if base == "height" else configs.jet_vortex
    members = [make(nx=24, ny=22, nz=nz, seed=5), make(nx=33, ny=19, nz=nz, seed=6, noise=0.2)]
    ens = anelastic.Ensemble(members, precision)
    for m, wl in enumerate(members):
        ens.load_member(m, wl.fields)
    if tune:
        ens.tune()
    ens.step(3)
    for m, wl in enumerate(members):
        solo = anelastic.Model(wl, precision)
        solo.step(3)
        for f in range(4):
            for slot in (abi.GA_SLOT_CUR, abi.GA_SLOT_P, abi.GA_SLOT_M):
                np.testing.assert_array_equal(ens.get(m, f, slot), solo.get(f, slot), err_msg=f"member {m} f{f} s{slot}")
        np.testing.assert_array_equal(ens.get(m, abi.GA_PI), solo.get(abi.GA_PI))
        solo.close()
    ens.close()
