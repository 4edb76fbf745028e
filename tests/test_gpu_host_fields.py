"""Host fields that abut in memory without being one allocation: a program may page-lock
its arrays one by one, or only some of them.  Transfers in both directions take them like
any other arrays, on both lanes."""
import ctypes as C
import mmap

import numpy as np
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from tests.helpers import CHECK_FIELDS, bitwise_equal, seeded_case, valid_mask

pytestmark = pytest.mark.gpu

ALIGN = 1 << 16  # the largest page size of the machines this runs on


class Fields:
    """n abutting arrays of `count` doubles in one anonymous mapping, those in `locked`
    page-locked by a call of their own (whole pages each)."""

    def __init__(self, n, count, locked):
        assert count * 8 % ALIGN == 0
        self.torch = pytest.importorskip("torch")
        self.torch.zeros(1, device="cuda")
        self.buf = mmap.mmap(-1, n * count * 8 + ALIGN)
        raw = np.frombuffer(self.buf, dtype=np.uint8)
        off = (-raw.ctypes.data) % ALIGN
        self.a = raw[off:off + n * count * 8].view(np.float64).reshape(n, count)
        self.locked = []
        for q in locked:
            rc = self.torch.cuda.cudart().cudaHostRegister(self.a[q].ctypes.data, count * 8, 0)
            assert int(rc) == 0
            self.locked.append(q)

    def release(self):
        for q in self.locked:
            self.torch.cuda.cudart().cudaHostUnregister(self.a[q].ctypes.data)


# none, one in the middle of a run, some, each by itself
@pytest.mark.parametrize("locked", [(), (1,), (0, 2, 3, 7), tuple(range(8))], ids=["none", "one", "some", "each"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_abutting_fields_page_locked_one_by_one(precision, locked):
    mesh, s, dt = seeded_case(58, 3, seed=3)  # (nh = 64: a field is 192 KiB, three 64 KiB pages)
    kw = dict(precision=precision, phi_mean=8000.0 * mesh.gravity)
    ref = M.Stepper(mesh, dt, **kw)
    ref.set_state(s)
    tend = ref.spatial_operator()
    ref.step(2)
    want = ref.get_state()
    m, im = valid_mask(mesh), mesh.interior_mask()
    F = Fields(9, mesh.ncell, locked)
    try:
        st = M.State({k: F.a[q] for q, k in enumerate(L.STATE_FIELDS)})
        for k in L.STATE_FIELDS:
            st[k][:] = s[k]
        g = M.Stepper(mesh, dt, **kw)
        g.set_state(st)
        g.step(2)
        g.get_state(st)
        for k in CHECK_FIELDS:
            assert bitwise_equal(st[k], want[k], m), k
        # the asynchronous calls, then the tendency into abutting arrays
        for k in L.STATE_FIELDS:
            st[k][:] = s[k]
        g.set_state_async(st)
        g.sync()
        ptr = [F.a[q].ctypes.data_as(C.POINTER(C.c_double)) for q in range(3)]
        L.check(L.lib().ccs_spatial_operator(g.handle, *ptr), "ccs_spatial_operator", g.handle)
        for q in range(3):
            assert bitwise_equal(F.a[q], tend[q], im), q
        g.step_async(2)
        g.get_state_async(st)
        g.sync()
        for k in CHECK_FIELDS:
            assert bitwise_equal(st[k], want[k], m), k
        g.close()
    finally:
        F.release()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_refused_transfer_leaves_no_error_behind(precision):
    """A field of which only a part is page-locked is refused by CUDA; the handle, and
    handles made after it, work on."""
    mesh, s, dt = seeded_case(58, 3, seed=4)
    kw = dict(phi_mean=8000.0 * mesh.gravity)
    F = Fields(1, mesh.ncell, ())
    rt = F.torch.cuda.cudart()
    assert int(rt.cudaHostRegister(F.a.ctypes.data, ALIGN, 0)) == 0  # the first third
    try:
        bad = M.State(dict(s.copy().arrays, u=F.a[0]))
        F.a[0][:] = s["u"]
        g = M.Stepper(mesh, dt, precision=precision, **kw)
        g.set_state(s)
        for again in ("fp64", "mixed"):
            with pytest.raises(L.CCSError):
                g.set_state(bad)
            h = M.Stepper(mesh, dt, precision=again, **kw)
            h.set_state(s)
            h.step(1)
            with pytest.raises(L.CCSError):
                g.get_state(bad)
            g.set_state(s)
            g.step(1)
            assert g.check_state() == 0 and h.check_state() == 0
    finally:
        rt.cudaHostUnregister(F.a.ctypes.data)
