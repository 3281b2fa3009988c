"""The pressure solve over transform lengths and level counts.

The y transform packs two levels into one complex line and keeps half of the
spectrum; the transforms run radix 8, 4, 2, 3 and 5 passes and one for any
other prime.  Each size here puts another radix, parity of the line length or
parity of the level count first.  The bounds are the parity tests' 1e-12 in
FP64 and 1e-5 in FP32, plus a unit roundoff times the condition of the
longest wave's vertical system, (L / (pi dz))^2 for a domain of length L.
"""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(12, 12, 6), (16, 13, 7), (17, 16, 8), (64, 24, 9), (30, 45, 12), (25, 64, 13), (49, 22, 10), (38, 128, 21),
         (27, 77, 16), (121, 33, 11), (512, 14, 33)]


@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_solve_pressure_sizes(size, periodic):
    nx, ny, nz = size
    nx += 6 * periodic  # the spectral grid of a periodic domain leaves the copied columns out
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dz=500.0, periodic=periodic)
    cols = anelastic.build_columns(wl)
    n3 = (nx, ny, nz)
    rnd = [2.0 * configs.splitmix_uniform(9100 + f, wl.points).reshape(n3) - 1.0 for f in range(3)]
    ref = O.Oracle(wl, cols)
    models = [anelastic.Model(wl, prec, columns=cols) for prec in (abi.GA_PREC_F64, abi.GA_PREC_F32)]
    for f, amp in ((abi.GA_U, 3.0), (abi.GA_V, 3.0), (abi.GA_W, 0.5)):
        for m in [ref] + models:
            m.set(f, abi.GA_SLOT_P, amp * rnd[f])
    ref.op("solve_pressure", 0.5)
    want = ref.get(abi.GA_PI)
    cond = (max(nx, ny) * wl.dx / (np.pi * wl.dz)) ** 2
    for m, tol in zip(models, (1e-12 + 2.0 ** -53 * cond, 1e-5 + 2.0 ** -24 * cond)):
        m.solve_pressure(0.5)
        got = m.get(abi.GA_PI)
        m.close()
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
