"""The marching FP32 advection kernel (k_advect_march) against the per-level
tile kernel (k_advect_tile): both evaluate the same face and tendency
expressions, so every advection operator agrees bit for bit.  The sizes put
the edges of its tiles first: the smallest grid, one thread row left over,
chunks of one column, few and many level quads.
"""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu

FIELDS = {"advect_uvw": (0, 1, 2), "advect_theta": (3,), "advect_micro": (4, 5, 6, abi.GA_VT)}


def _models(monkeypatch, wl):
    ms = []
    for mode in ("tile", "march"):
        monkeypatch.setenv("GA_ADVECT", mode)
        ms.append(anelastic.Model(wl, abi.GA_PREC_F32))
    monkeypatch.delenv("GA_ADVECT")
    return ms


def _perturb(ms, wl, seed):
    rng = np.random.default_rng(seed)
    for f, scale in enumerate([2.0, 2.0, 0.5, 0.3, 1e-3, 4e-4, 4e-4][: 7 if wl.microphysics_option else 4]):
        for slot in (abi.GA_SLOT_CUR, abi.GA_SLOT_M):
            x = rng.standard_normal(wl.points) * scale + (2e-4 if f >= 5 else 0.0)
            x[rng.random(wl.points) < 0.1] = 0.0
            for m in ms:
                m.set(f, slot, x)


@pytest.mark.parametrize("kind", ["rf1", "rf2", "dry", "periodic"])
@pytest.mark.parametrize("size", [(12, 12, 8), (13, 41, 24), (47, 12, 32), (40, 37, 48), (24, 30, 128)],
                         ids=lambda s: "x".join(map(str, s)))
def test_operators_bit_identical(monkeypatch, kind, size):
    nx, ny, nz = size
    if kind == "dry":
        wl = configs.dry_bubble(nx=nx, ny=ny, nz=nz)
    else:
        wl = configs.moist_blob(nx=nx + 6 * (kind == "periodic"), ny=ny, nz=nz, dz=200.0 if nz > 64 else 400.0,
                                rain_fallout=2 if kind == "rf2" else 1, periodic=int(kind == "periodic"))
    ms = _models(monkeypatch, wl)
    _perturb(ms, wl, 31)
    for op, fields in FIELDS.items():
        if op == "advect_micro" and kind == "dry":
            continue
        for m in ms:
            m.op(op, 0.5)
        for f in fields:
            a, b = (m.get(f, abi.GA_SLOT_P) for m in ms)
            np.testing.assert_array_equal(b, a, err_msg=f"{kind} {op} field {f}")


@pytest.mark.parametrize("kind", ["kessler", "adjoint"])
def test_steps_bit_identical(monkeypatch, kind):
    """whole steps: every slot, and a gradient, whose forward run records the
    clipped points through the marching kernel's combined moisture job"""
    wl = configs.moist_blob(nx=33, ny=29, nz=20)
    ms = _models(monkeypatch, wl)
    if kind == "adjoint":
        rng = np.random.default_rng(5)
        seed = rng.random(wl.points) - 0.5
        for m in ms:
            for f in m.lin_fields():
                m.lin_set(f, abi.GA_SLOT_CUR, seed)
            m.adjoint(3, 2)
        for k, v in ms[0].lin_get_all().items():
            np.testing.assert_array_equal(ms[1].lin_get(*k), v, err_msg=str(k))
    else:
        for m in ms:
            m.step(3)
        a, b = (m.state() for m in ms)
        for k in a:
            np.testing.assert_array_equal(b[k], a[k], err_msg=k)
