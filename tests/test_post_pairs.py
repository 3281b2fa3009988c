"""The FP64 column pass on pairs of levels (k_post_quad) against the column
kernel (GA_POST=column): the same expressions without contraction, so whole
steps agree bit for bit.  Level counts at the ends of the range and one that
is not a multiple of four; a sponge, a periodic domain, the ice scheme's
second pass."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["moist", "periodic", "dry", "ice"])
@pytest.mark.parametrize("nz", [6, 18, 128])
def test_steps_bit_identical(monkeypatch, kind, nz):
    if kind == "dry":
        wl = configs.dry_bubble(nx=19, ny=17, nz=nz)
    elif kind == "ice":
        wl = configs.ice_cloud(nx=19, ny=17, nz=nz, dz=200.0 if nz > 64 else 600.0)
    else:
        wl = configs.moist_blob(nx=19, ny=17, nz=nz, dz=200.0 if nz > 64 else 500.0, periodic=int(kind == "periodic"))
    ms = []
    for mode in ("column", "quad"):
        monkeypatch.setenv("GA_POST", mode)
        ms.append(anelastic.Model(wl, abi.GA_PREC_F64))
    for m in ms:
        m.step(2)
    a, b = (m.state() for m in ms)
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)
