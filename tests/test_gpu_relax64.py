"""The FP64 relaxation's launch shapes (lanes per column, warps per column)
against the oracle, bit for bit: LJ and Coulomb scans whose column counts
reach every shape and whose atom counts lie around the rounds and passes of
the terms.  Scans over an external field or a rigid grid, where the oracle
agrees to rounding only, are compared between shapes."""
import numpy as np
import pytest

import oracle
from mechafm_gb300 import _abi, synth
from mechafm_gb300.scan import Input, Scan

pytestmark = pytest.mark.gpu


def molecule(tmp_path, atoms, nx, ny, **opt):
    spec = synth.molecule_batch(1, seed=atoms + nx, grids=(8,), atoms=(atoms, atoms), zlow=9.85, **opt)[0]
    spec.options["area"] = f"{0.1 * (nx - 1) + 1e-6!r} {0.1 * (ny - 1) + 1e-6!r}"
    d = Input(spec.write(str(tmp_path))).desc()
    assert d.shape[:2] == (nx, ny) and d.c.n_atoms == atoms
    return d


def same(got, want):
    for key in ("steps", "tip", "force", "energy"):
        np.testing.assert_array_equal(got[key], want[key], err_msg=key)


@pytest.mark.parametrize("atoms,nx,ny,opt", [
    (1, 3, 2, {}), (15, 5, 1, {}),                     # too few terms for several warps
    (16, 1, 1, {}), (31, 3, 3, {}), (32, 2, 2, {}),    # one warp's chunk of terms and the tip-dummy term
    (127, 3, 2, {}), (128, 2, 2, {}), (200, 2, 2, {"integrator": "rk4"}),   # passes of the terms
    (20, 35, 31, {}), (33, 36, 31, {"coulomb": "off"}),   # past the last column of the several-warp shape
    (20, 44, 30, {"integrator": "euler"}),             # 16 lanes
    (21, 51, 50, {}), (20, 49, 51, {"minimiser": "SD", "maxsteps": "40"}),   # 8 lanes
    (17, 71, 70, {}), (20, 70, 71, {"coulomb": "off", "integrator": "rk4"}),  # 4 lanes
])
def test_every_shape_has_the_oracles_bits(tmp_path, atoms, nx, ny, opt):
    d = molecule(tmp_path, atoms, nx, ny, **opt)
    want, steps = oracle.run(d)
    scan = Scan(d, device=0)
    got, st = scan.run(_abi.FP64)
    same(got, want)
    assert st.total_steps == steps == int(got["steps"].sum())
    # a range of columns, and chosen columns in any order, are the same points
    n, nz = d.n_columns, d.c.nz
    b, e = n // 3, n // 3 + max(1, n // 2)
    part, _ = scan.run(_abi.FP64, col_begin=b, col_end=e)
    same(part, want[b * nz:e * nz])
    cols = np.random.default_rng(atoms).permutation(n)[:min(n, 40)]
    chosen, _ = scan.run_columns(cols)
    same(chosen.reshape(len(cols), nz), want.reshape(n, nz)[cols])


@pytest.mark.parametrize("rigid", [False, True])
@pytest.mark.parametrize("pixels", [36, 50, 70])
def test_field_and_grid_shapes_agree(tmp_path, rigid, pixels):
    spec = synth.slab(seed=3, nlx=4, nly=4, layers=2, cell=(10.0, 10.0, 20.0), cube_n=(40, 40, 80), pixels=pixels,
                      step=0.15, zhigh=18.0, zlow=17.85, rigidgrid=rigid, tip_charge=-0.02, vdw_pbc="off")
    scan = Scan(Input(spec.write(str(tmp_path))).desc(), device=0)
    got, st = scan.run(_abi.FP64)
    n, nz = scan.desc.n_columns, scan.desc.c.nz
    assert st.error_word & ~_abi.PT_MAXSTEPS == 0
    for b in range(0, n, 300):
        part, _ = scan.run_columns(np.arange(b, min(n, b + 300)))
        np.testing.assert_array_equal(part, got[b * nz:(b + len(part) // nz) * nz])
