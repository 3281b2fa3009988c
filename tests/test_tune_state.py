"""The autotuner leaves the state as it was, in every set of equations: all
slots, pi and the fall speeds, bit for bit (the hydrostatic set's w lives in
its current slot, which the timed kernels take for the forecast one)."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.GA_PREC_F64, abi.GA_PREC_F32], ids=["f64", "f32"])
@pytest.mark.parametrize("kind", ["dry", "moist", "periodic", "ice", "linear", "hydrostatic_dry", "hydrostatic_moist",
                                  "hydrostatic_ice", "physics"])
def test_state_unchanged(kind, precision):
    k = dict(nx=26, ny=23, nz=16)
    if kind.endswith("dry"):
        wl = configs.dry_bubble(**k)
    elif kind.endswith("ice"):
        wl = configs.ice_cloud(**k)
    else:
        wl = configs.moist_blob(periodic=int(kind == "periodic"), **k)
    if kind.startswith("hydrostatic"):
        wl.hydrostatic, wl.dt = 1, 2.0
    wl.linear_model = int(kind == "linear")
    if kind == "physics":
        wl.use_explicit_diffusion, wl.turbulence_option, wl.use_surface_heat_flux = 1, 1, 1
    m = anelastic.Model(wl, precision)
    m.step(2)
    before = m.state()
    m.tune()
    after = m.state()
    for f in before:
        np.testing.assert_array_equal(after[f], before[f], err_msg=f)
