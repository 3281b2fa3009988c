"""The paired fused x kernel (GA_SPECTRAL_X=pair) on lines whose default block
would have more threads than its registers allow.  The default block grows
with the line and the level count; the paired kernel computes the same
columns, so whole steps agree bit for bit."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


# default blocks of 512, 736, 992 and 988 threads
@pytest.mark.parametrize("size", [(64, 22, 66), (128, 20, 48), (128, 24, 64), (203, 18, 40)],
                         ids=lambda s: "x".join(map(str, s)))
def test_pair_matches_single_block(monkeypatch, size):
    nx, ny, nz = size
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dz=300.0)
    ms = []
    for mode in ("single", "pair"):
        monkeypatch.setenv("GA_SPECTRAL_X", mode)
        ms.append(anelastic.Model(wl, abi.GA_PREC_F32))
    monkeypatch.delenv("GA_SPECTRAL_X")
    for m in ms:
        m.step(3)
    a, b = (m.state() for m in ms)
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)
