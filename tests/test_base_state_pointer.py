"""A basic state written through its device pointer (ga_field_device_ptr): the
next step reads it, as after ga_set_field.  FP64 contexts on a basic state
that varies horizontally keep faces of it; the pointer may be asked for before
the first step or after it."""
import numpy as np
import pytest

from model_gb300 import abi, anelastic, configs

pytestmark = pytest.mark.gpu


class _Array:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


@pytest.mark.parametrize("when", ["before", "after"])
@pytest.mark.parametrize("precision", [abi.GA_PREC_F64, abi.GA_PREC_F32], ids=["f64", "f32"])
@pytest.mark.parametrize("moist", [False, True])
def test_written_pointer_equals_set_field(moist, precision, when):
    torch = pytest.importorskip("torch")
    wl = configs.jet_vortex(nx=26, ny=22, nz=12, moist=moist, extra_basic=0.3)
    a, b = anelastic.Model(wl, precision), anelastic.Model(wl, precision)
    bars = {abi.GA_UBAR: "ubar", abi.GA_VBAR: "vbar", abi.GA_THBAR: "thbar"}
    if moist:
        bars[abi.GA_QBAR] = "qbar"
    ptrs = {f: b.device_ptr(f) for f in bars} if when == "before" else {}
    for m in (a, b):
        m.step(2)  # (the captured graph holds the faces too)
    real = np.float64 if precision == abi.GA_PREC_F64 else np.float32
    for f, name in bars.items():
        new = (1.25 * wl.fields[name]).ravel()
        a.set(f, 0, new)
        dst = torch.as_tensor(_Array(ptrs.get(f) or b.device_ptr(f), new.size, np.dtype(real).str), device="cuda")
        dst.copy_(torch.from_numpy(new.astype(real)))
    torch.cuda.synchronize()
    for m in (a, b):
        m.step(2)
    x, y = a.state(), b.state()
    for k in x:
        np.testing.assert_array_equal(y[k], x[k], err_msg=k)
