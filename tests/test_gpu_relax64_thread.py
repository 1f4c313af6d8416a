"""The FP64 relaxation with one thread a column (many columns, few terms) against the
oracle, bit for bit, with column counts on both sides of the rule (152 SMs times
110 columns, 400 from 11 terms on); over an external field or a rigid grid, where the
oracle agrees to rounding only, against calls of few columns, which take lanes."""
import numpy as np
import pytest

import oracle
from mechafm_gb300 import _abi, synth
from mechafm_gb300.scan import Input, Scan
from test_gpu_relax64 import molecule, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,nx,ny,opt", [
    (1, 152, 110, {"coulomb": "off"}), (1, 5573, 3, {"coulomb": "off"}),   # 16,720 columns and one fewer
    (4, 152, 110, {}), (10, 131, 128, {"integrator": "rk4"}), (11, 152, 110, {}),
    (6, 131, 128, {"integrator": "euler"}), (5, 150, 112, {"minimiser": "SD", "maxsteps": "30"}),
    (4, 149, 113, {"minterm": "e"}), (7, 149, 113, {"minterm": "f", "coulomb": "off"}),
    (20, 304, 200, {"maxsteps": "20"}), (20, 267, 227, {"maxsteps": "20"}),   # 60,800 and 191 fewer
])
def test_one_thread_has_the_oracles_bits(tmp_path, atoms, nx, ny, opt):
    d = molecule(tmp_path, atoms, nx, ny, **opt)
    want, steps = oracle.run(d)
    scan = Scan(d, device=0)
    got, st = scan.run(_abi.FP64)
    same(got, want)
    assert st.total_steps == steps == int(got["steps"].sum())
    n, nz = d.n_columns, d.c.nz
    part, few = scan.run(_abi.FP64, col_begin=17, col_end=317)   # lanes
    same(part, want[17 * nz:317 * nz])
    again, many = scan.run(_abi.FP64, col_begin=1, col_end=n)
    same(again, want[nz:])
    assert many.pair_evals * few.force_evals == few.pair_evals * many.force_evals
    cols = np.random.default_rng(atoms).permutation(n)
    chosen, _ = scan.run_columns(cols)
    same(chosen.reshape(n, nz), want.reshape(n, nz)[cols])


@pytest.mark.parametrize("rigid,zhigh,pixels,opt", [
    (False, 14.0, 130, {}), (True, 14.0, 86, {}), (True, 14.0, 86, dict(integrator="rk4")),
    (False, 14.0, 131, dict(integrator="euler")),
    (False, 7.2, 199, {}), (True, 7.2, 124, {}),   # the tip within 3.5 A of the atoms
])
def test_field_and_grid_agree_with_calls_of_few_columns(tmp_path, rigid, zhigh, pixels, opt):
    spec = synth.slab(seed=3, nlx=2, nly=2, layers=1, cell=(10.0, 10.0, 20.0), cube_n=(40, 40, 80), pixels=pixels,
                      step=0.05, zhigh=zhigh, zlow=zhigh - 0.15, rigidgrid=rigid, tip_charge=-0.02, vdw_pbc="off", **opt)
    scan = Scan(Input(spec.write(str(tmp_path))).desc(), device=0)
    got, st = scan.run(_abi.FP64)
    n, nz = scan.desc.n_columns, scan.desc.c.nz
    assert st.error_word & ~_abi.PT_MAXSTEPS == 0
    for b in range(0, n, 2000):
        part, _ = scan.run_columns(np.arange(b, min(n, b + 300)))
        same(part, got[b * nz:(b + len(part) // nz) * nz])
