"""FP32 of two solves against the oracle: the hydrostatic lid pressure over
line lengths, and the semi-Lagrangian rain fallout.  The bounds are the parity
tests' 1e-5, for the lid plus a unit roundoff times the condition of the
longest wave's system, (n / pi)^2 for n points."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(12, 12, 6), (13, 30, 9), (50, 17, 16), (33, 64, 33), (128, 128, 8)],
                         ids=lambda s: "x".join(map(str, s)))
def test_hydrostatic_lid(size):
    nx, ny, nz = size
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dx=2000.0)
    wl.hydrostatic = 1
    rng = np.random.default_rng(29)
    cols = anelastic.build_columns(wl)
    m, o = anelastic.Model(wl, abi.GA_PREC_F32, columns=cols), O.Oracle(wl, cols)
    for f in (abi.GA_U, abi.GA_V):
        x = rng.standard_normal(wl.points).astype(np.float32)
        for a in (m, o):
            a.set(f, abi.GA_SLOT_P, x)
    for a in (m, o):
        a.op("solve_pressure", 0.5)
    got, want = m.get(abi.GA_PI), o.get(abi.GA_PI)
    tol = 1e-5 + 2.0 ** -24 * (max(nx, ny) / np.pi) ** 2
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("rain", ["top_everywhere", "top_in_patches", "below"])
@pytest.mark.parametrize("size", [(12, 13, 6), (41, 30, 33), (20, 21, 128)], ids=lambda s: "x".join(map(str, s)))
def test_fallout(size, rain):
    nx, ny, nz = size
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dz=150.0 if nz > 64 else 400.0, rain_fallout=2)
    rng = np.random.default_rng(31)
    qr = 1e-3 * rng.random((nx, ny, nz), dtype=np.float32)
    if rain == "below":
        qr[:, :, nz // 2:] = 0.0
    elif rain == "top_in_patches":
        qr[rng.random((nx, ny)) < 0.6, nz // 2:] = 0.0
        qr[rng.random((nx, ny)) < 0.3] = 0.0
    cols = anelastic.build_columns(wl)
    m, o = anelastic.Model(wl, abi.GA_PREC_F32, columns=cols), O.Oracle(wl, cols)
    for x in (m, o):
        x.set(abi.GA_TH, abi.GA_SLOT_P, wl.fields["th"])
        x.set(abi.GA_QV, abi.GA_SLOT_P, wl.fields["qv"])
        x.set(abi.GA_QR, abi.GA_SLOT_P, qr)
        for _ in range(2):
            x.op("kessler")
    for f, slot in ((abi.GA_QR, abi.GA_SLOT_P), (abi.GA_ACCRAIN, 0)):
        a, b = m.get(f, slot), o.get(f, slot)
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
