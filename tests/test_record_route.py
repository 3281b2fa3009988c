"""Recorded (linearised) moist FP32 steps take the four-level tile kernel on
small flat grids and the marching kernel elsewhere: gradients and tangents are
the same bit for bit as with either kernel alone, on both sides of the line."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(16, 18, 8), (26, 23, 32), (26, 23, 36), (101, 94, 32)],
                         ids=lambda s: "x".join(map(str, s)))
def test_default_equals_each_kernel(monkeypatch, size):
    nx, ny, nz = size
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dz=400.0)
    rng = np.random.default_rng(8)
    seed = rng.standard_normal(wl.points)
    out = []
    for mode in ("default", "march", "quad"):
        monkeypatch.setenv("GA_ADVECT", mode)
        m = anelastic.Model(wl, abi.GA_PREC_F32)
        monkeypatch.delenv("GA_ADVECT")
        for f in m.lin_fields():
            m.lin_set(f, abi.GA_SLOT_CUR, seed)
        m.adjoint(3, 2)
        res = m.lin_get_all()
        m.tlm_step(1)
        res.update({("tlm",) + k: v for k, v in m.lin_get_all().items()})
        out.append(res)
        m.close()
    for k, v in out[0].items():
        for other in out[1:]:
            np.testing.assert_array_equal(other[k], v, err_msg=str(k))
