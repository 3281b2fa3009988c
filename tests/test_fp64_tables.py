"""FP64 contexts without the tables they can do without (GA_FP64_TABLES=0, or
no room for them): the same results bit for bit as with them, in steps,
gradients and ensembles, and the memory of a context without them."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu

KINDS = ["moist", "periodic", "jet", "jet_moist", "linear", "hydrostatic"]


def _wl(kind, nx=26, ny=22, nz=13):
    if kind.startswith("jet") or kind == "linear":
        wl = configs.jet_vortex(nx=nx, ny=ny, nz=nz, moist=kind == "jet_moist", extra_basic=0.3, noise=0.1)
        wl.linear_model = int(kind == "linear")
        return wl
    wl = configs.moist_blob(nx=nx + 6 * (kind == "periodic"), ny=ny, nz=nz, periodic=int(kind == "periodic"))
    if kind == "hydrostatic":
        wl.hydrostatic, wl.dt = 1, 2.0
    return wl


def _both(monkeypatch, make):
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("GA_FP64_TABLES", on)
        out.append(make())
    monkeypatch.delenv("GA_FP64_TABLES")
    return out


@pytest.mark.parametrize("kind", KINDS)
def test_steps(monkeypatch, kind):
    ms = _both(monkeypatch, lambda: anelastic.Model(_wl(kind), abi.GA_PREC_F64))
    for m in ms:
        m.step(3)
    a, b = (m.state() for m in ms)
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)


@pytest.mark.parametrize("kind", ["moist", "jet"])
def test_gradients(monkeypatch, kind):
    ms = _both(monkeypatch, lambda: anelastic.Model(_wl(kind), abi.GA_PREC_F64))
    seed = np.random.default_rng(4).standard_normal(ms[0].n3)
    for m in ms:
        for f in m.lin_fields():
            m.lin_set(f, abi.GA_SLOT_CUR, seed)
        m.adjoint(3, 2)
    a, b = (m.lin_get_all() for m in ms)
    for k in a:
        np.testing.assert_array_equal(b[k], a[k], err_msg=str(k))


def test_ensemble(monkeypatch):
    wls = [_wl("jet"), _wl("jet", 33, 19, 16)]
    es = _both(monkeypatch, lambda: anelastic.Ensemble(wls, abi.GA_PREC_F64))
    for e in es:
        for m, wl in enumerate(wls):
            e.load_member(m, wl.fields)
        e.step(3)
    for m in range(len(wls)):
        for f in range(4):
            np.testing.assert_array_equal(es[1].get(m, f), es[0].get(m, f))


def test_memory(monkeypatch):
    torch = pytest.importorskip("torch")
    wl = _wl("jet", 128, 96, 32)
    used = []

    def make():
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        m = anelastic.Model(wl, abi.GA_PREC_F64)
        m.step(2)
        torch.cuda.synchronize()
        used.append(free - torch.cuda.mem_get_info()[0])
        return m
    make().close()  # (what the first context of a process loads)
    used.clear()
    for m in _both(monkeypatch, make):
        m.close()
    assert used[0] - used[1] > 15 * 8 * wl.points  # the faces of three fields
