"""The FP64 relaxation with one thread a column (many columns, few terms) against the
oracle, bit for bit, with column counts on both sides of the rule (152 SMs times
45 columns and 4 or 10 more per term); over an external field or a rigid grid,
where the oracle agrees to rounding only, against calls of few columns."""
import numpy as np
import pytest

import oracle
from mechafm_gb300 import _abi, synth
from mechafm_gb300.scan import Input, Scan
from test_gpu_relax64 import molecule, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,nx,ny,opt", [
    (1, 88, 95, {"coulomb": "off"}), (1, 643, 13, {"coulomb": "off"}),   # 8,360 columns and one fewer
    (4, 76, 122, {}), (4, 843, 11, {"integrator": "rk4"}),               # 9,272, and one more
    (6, 107, 106, {"integrator": "euler"}), (5, 120, 101, {"minimiser": "SD", "maxsteps": "30"}),
    (4, 131, 120, {"minterm": "e"}), (7, 150, 123, {"minterm": "f", "coulomb": "off"}),
    (114, 279, 278, {"maxsteps": "4"}),                                  # blocks of 128 threads
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


@pytest.mark.parametrize("rigid,opt", [(False, {}), (True, {}), (True, dict(integrator="rk4")), (False, dict(integrator="euler"))])
def test_field_and_grid_agree_with_calls_of_few_columns(tmp_path, rigid, opt):
    spec = synth.slab(seed=3, nlx=2, nly=2, layers=1, cell=(10.0, 10.0, 20.0), cube_n=(40, 40, 80), pixels=117,
                      step=0.05, zhigh=14.0, zlow=13.85, rigidgrid=rigid, tip_charge=-0.02, vdw_pbc="off", **opt)
    scan = Scan(Input(spec.write(str(tmp_path))).desc(), device=0)
    got, st = scan.run(_abi.FP64)
    n, nz = scan.desc.n_columns, scan.desc.c.nz
    assert n >= 152 * (45 + 10 * scan.desc.c.n_atoms) and st.error_word & ~_abi.PT_MAXSTEPS == 0
    for b in range(0, n, 900):
        part, _ = scan.run_columns(np.arange(b, min(n, b + 300)))
        same(part, got[b * nz:(b + len(part) // nz) * nz])
