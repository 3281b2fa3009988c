"""Semi-Lagrangian rain fallout against the oracle: the edge value carried
between rainy columns, which one block starts anywhere a column forgets its
past or, with no such column near, walks in order.  Rain up to the top level
in every column (nothing forgets), in patches, and nowhere near the top; level
counts at the ends of the range.  The bound is the parity tests' 1e-12."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rain", ["top_everywhere", "top_in_patches", "below"])
@pytest.mark.parametrize("size", [(12, 13, 6), (41, 30, 33), (20, 21, 128)], ids=lambda s: "x".join(map(str, s)))
def test_fallout(size, rain):
    nx, ny, nz = size
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dz=150.0 if nz > 64 else 400.0, rain_fallout=2)
    rng = np.random.default_rng(17)
    qr = 1e-3 * rng.random((nx, ny, nz))
    if rain == "below":
        qr[:, :, nz // 2:] = 0.0
    elif rain == "top_in_patches":
        qr[rng.random((nx, ny)) < 0.6, nz // 2:] = 0.0
        qr[rng.random((nx, ny)) < 0.3] = 0.0
    cols = anelastic.build_columns(wl)
    m, o = anelastic.Model(wl, abi.GA_PREC_F64, columns=cols), O.Oracle(wl, cols)
    for x in (m, o):
        x.set(abi.GA_TH, abi.GA_SLOT_P, wl.fields["th"])
        x.set(abi.GA_QV, abi.GA_SLOT_P, wl.fields["qv"])
        x.set(abi.GA_QR, abi.GA_SLOT_P, qr)
        for _ in range(2):  # the carried value runs on into the next call
            x.op("kessler")
    for f, slot in ((abi.GA_QR, abi.GA_SLOT_P), (abi.GA_ACCRAIN, 0)):
        a, b = m.get(f, slot), o.get(f, slot)
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
