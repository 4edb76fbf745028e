"""Run in a process that loaded the bounds-checked library (CCS_GPU_LIB): both lanes, every
variant and option on small grids, on which that build runs every tile and part shape of
both lanes.  Exits non-zero at the first recorded out-of-range index; prints the shapes it
met, lane by lane."""
import ctypes as C
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

from conformal_cubed_sphere_gb300 import _lib as L  # noqa: E402
from conformal_cubed_sphere_gb300 import model as M  # noqa: E402

# (N, halo): one tile and several, partial ones, halos from 3 to the panel width
GRIDS = [(4, 3), (6, 6), (13, 4), (20, 4), (33, 3), (40, 5), (50, 3), (66, 4)]
OPTIONS = [("RK4", L.CCS_EDISS_ZERO, L.CCS_OP_WENO), ("RK4", L.CCS_EDISS_RECONSTRUCT, L.CCS_OP_WENO),
           ("RK3_TVD", L.CCS_EDISS_ZERO, L.CCS_OP_WENO), ("RK3_TVD", L.CCS_EDISS_RECONSTRUCT, L.CCS_OP_WENO),
           ("RK4", L.CCS_EDISS_ZERO, L.CCS_OP_CENTRAL4), ("RK3_TVD", L.CCS_EDISS_ZERO, L.CCS_OP_CENTRAL6)]


def grid_state(N, halo):
    mesh = M.Mesh(N, halo, pole_inverse=N % 2 == 1)
    s = M.initial_state(mesh, kind=L.CCS_IC_SEEDED, seed=N, lmax_oro=8)
    return mesh, s, M.cfl_dt(mesh, s, 0.5)


def runs(grids):
    """(key, tile shape, tendencies, state) of every case"""
    for N, halo in grids:
        mesh, s, dt = grid_state(N, halo)
        for lane, nvar in (("fp64", 3), ("mixed", len(L.MIXED_VARIANTS))):
            for var in range(nvar):
                for opt, (scheme, ediss, op) in enumerate(OPTIONS):
                    g = M.Stepper(mesh, dt, precision=lane, scheme=scheme, e_dissipation=ediss, operator=op,
                                  phi_mean=8000.0 * mesh.gravity)
                    g.set_variant(var)
                    g.set_state(s)
                    tend = g.spatial_operator()
                    g.step(2)
                    nbad = g.check_state()
                    if nbad:  # (the checked build poisons shared arrays with NaN)
                        raise SystemExit(f"C{N} {lane} variant {var} option {opt}: {nbad} bad cells")
                    yield (N, halo, lane, var, opt), g.stage_tile[:2], tend, g.get_state()
                    g.close()


def main():
    if not str(L.LIB_PATH).endswith("bounds/libccs_gpu.so"):
        raise SystemExit(f"not the bounds-checked library: {L.LIB_PATH}")
    shapes = {"fp64": set(), "mixed": set()}
    site, idx = C.c_int(0), C.c_int64(0)
    for key, tile, _, _ in runs(GRIDS):
        L.check(L.lib().ccs_debug_bounds(C.byref(site), C.byref(idx)), "ccs_debug_bounds")
        if site.value:
            raise SystemExit(f"{key}: out-of-range index {idx.value} at check site {site.value}")
        shapes[key[2]].add(tile + (key[4],))
    for lane, seen in shapes.items():
        for x, y, opt in sorted(seen):
            print("shape", lane, x, y, opt)


if __name__ == "__main__":
    main()
