"""Cell offsets are held in 32 bits: a grid whose field has 2^31 cells or more (a halo as
wide as a large panel) is refused before anything is read or allocated."""
import ctypes as C

import numpy as np
import pytest

from conformal_cubed_sphere_gb300 import _lib as L


@pytest.mark.parametrize("precision", [L.CCS_FP64, L.CCS_MIXED])
@pytest.mark.parametrize("N,halo", [(8192, 8192), (8192, 5400), (6400, 6400)])
def test_fields_of_2_to_the_31_cells_are_refused(precision, N, halo):
    assert 6 * (N + 2 * halo) ** 2 >= 2 ** 31
    cfg = L.Config(N=N, halo=halo, scheme=0, precision=precision, e_dissipation=0, device=0, dx=0.1, dy=0.1, dt=10.0,
                   radius=6.371e6, gravity=9.80616, omega=7.292e-5, phi_mean=0.0)
    one = np.zeros(1)  # (never read)
    ptr = one.ctypes.data_as(C.POINTER(C.c_double))
    mv = L.MeshView(**{k: ptr for k, _ in L.MeshView._fields_})
    h = C.c_void_p()
    assert L.lib().ccs_init(C.byref(cfg), C.byref(mv), C.byref(h)) == L.CCS_ERR_ARG
    assert not h.value
