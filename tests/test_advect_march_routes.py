"""The marching advection's other routes, bit for bit against the kernels that
do the same work apart: grids too large for L2 (three blocks an SM, the jobs of
a tile next to each other) against the tile kernel; snow and ice in the
moisture launch against the four-level tile kernel; the hydrostatic set's
lateral copies, made by the advection launch, against their own kernel."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


def _models(monkeypatch, wl, other):
    ms = []
    for mode in (other, "march"):
        monkeypatch.setenv("GA_ADVECT", mode)
        ms.append(anelastic.Model(wl, abi.GA_PREC_F32))
    monkeypatch.delenv("GA_ADVECT")
    return ms


def _same(ms):
    a, b = (m.state() for m in ms)
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)


# ten FP32 fields above 96 MiB; a row and a column of cells left over
@pytest.mark.parametrize("kind", ["moist", "dry"])
def test_large_grid(monkeypatch, kind):
    nx, ny, nz = 263, 245, 40
    wl = configs.moist_blob(nx=nx, ny=ny, nz=nz, dz=400.0) if kind == "moist" else \
        configs.dry_bubble(nx=nx, ny=ny, nz=nz)
    ms = _models(monkeypatch, wl, "tile")
    rng = np.random.default_rng(12)
    for f, s in ((abi.GA_U, 2.0), (abi.GA_V, 2.0), (abi.GA_W, 0.5)):
        x = s * rng.standard_normal(wl.points)
        for m in ms:
            m.set(f, abi.GA_SLOT_CUR, x)
    for m in ms:
        m.step(1)
    _same(ms)
    if kind == "moist":  # and with the clipping record (the three moisture fields in one job)
        seed = rng.standard_normal(wl.points)
        for m in ms:
            m.lin_set(abi.GA_QV, abi.GA_SLOT_CUR, seed)
            m.tlm_step(1)
        for f in ms[0].lin_fields():
            np.testing.assert_array_equal(ms[1].lin_get(f), ms[0].lin_get(f), err_msg=f"tangent {f}")


@pytest.mark.parametrize("rain_fallout", [1, 2])
@pytest.mark.parametrize("size", [(13, 41, 24), (24, 20, 16), (40, 37, 48)], ids=lambda s: "x".join(map(str, s)))
def test_snow_and_ice(monkeypatch, size, rain_fallout):
    nx, ny, nz = size
    wl = configs.ice_cloud(nx=nx, ny=ny, nz=nz, dz=450.0, rain_fallout=rain_fallout)
    ms = _models(monkeypatch, wl, "quad")
    for m in ms:
        m.step(3)
    _same(ms)


@pytest.mark.parametrize("kind", ["moist", "dry", "ice"])
def test_hydrostatic_copies(monkeypatch, kind):
    k = dict(nx=29, ny=33, nz=20)
    wl = configs.dry_bubble(**k) if kind == "dry" else configs.ice_cloud(**k) if kind == "ice" else configs.moist_blob(**k)
    wl.hydrostatic, wl.dt = 1, 2.0
    ms = _models(monkeypatch, wl, "quad" if kind == "ice" else "tile")
    for m in ms:
        m.step(3)
    _same(ms)
