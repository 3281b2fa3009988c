"""The lid-pressure solve of the hydrostatic set over line lengths: x lines of
every radix, wavenumber blocks with a remainder, and y lines too long for
shared memory.  FP64 against the oracle, the parity tests' 1e-12."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(12, 12, 6), (13, 30, 9), (50, 17, 16), (33, 64, 33), (12, 1700, 6)],
                         ids=lambda s: "x".join(map(str, s)))
def test_solve_pressure(size):
    nx, ny, nz = size
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dx=2000.0)
    wl.hydrostatic = 1
    rng = np.random.default_rng(23)
    cols = anelastic.build_columns(wl)
    m, o = anelastic.Model(wl, abi.GA_PREC_F64, columns=cols), O.Oracle(wl, cols)
    for f in (abi.GA_U, abi.GA_V):
        x = rng.standard_normal(wl.points)
        for a in (m, o):
            a.set(f, abi.GA_SLOT_P, x)
    for a in (m, o):
        a.op("solve_pressure", 0.5)
    got, want = m.get(abi.GA_PI), o.get(abi.GA_PI)
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
