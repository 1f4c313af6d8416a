"""The interpolated build of the double-float rigid grid: which scans take it,
and its nodes against the FP64 build where every term counts by itself, far
above the surface."""
import pytest

import numpy as np

from mechafm_gb300.scan import Input, Scan
from mechafm_gb300 import _abi, synth
from test_gpu_df_grid import SPECS, small_slab

pytestmark = pytest.mark.gpu


def _desc(spec, tmp_path):
    return Input(spec.write(str(tmp_path))).desc()


def _morse_slab(types):
    spec = small_slab(pixels=76, step=0.2, external=False, zhigh=26.0, zlow=25.85)
    spec.overwrites = [("O", t, "morse", 0.1, 1.5, 3.2) for t in types]
    return spec


ROUTES = dict(SPECS, morse_and_lj=lambda: _morse_slab(("C",)), morse=lambda: _morse_slab(("C", "N")),
              few_records=lambda: synth.cluster_60(n_atoms=124, area=7.9, step=0.1, zhigh=10.0, zlow=9.85,
                                                   coulomb="off", rigidgrid="on"))


@pytest.mark.parametrize("name", ROUTES)
def test_which_build_runs(tmp_path, name):
    scan = Scan(_desc(ROUTES[name](), tmp_path), device=0)
    _, blocks = scan.grid_df()
    assert (min(blocks) > 0) == (name not in ("sheared", "morse", "few_records")), blocks


HIGH = dict(zhigh=26.0, zlow=25.85)


def _lj_molecule():
    spec = synth.cluster_60(n_atoms=600, area=7.9, step=0.2, zhigh=18.0, zlow=17.85, coulomb="off", rigidgrid="on")
    spec.overwrites = []
    return spec


FAR = {"slab": lambda: small_slab(pixels=76, step=0.2, external=False, **HIGH), "molecule": _lj_molecule}


@pytest.mark.parametrize("attraction", [True, False])
@pytest.mark.parametrize("name", FAR)
def test_far_nodes_keep_their_relative_accuracy(tmp_path, name, attraction):
    """LJ terms only, all of one sign there.  A double-float term's force takes some
    16 operations of 2^-45 from its 1/r (4.5e-13), positions of 30 A to 2^-48 add
    1e-13 at 14 A, interpolation adds at most 3.1e-13 (a force r^-13 beside a thin
    block), and as much again for sums of a few thousand terms: below 2^-38."""
    d = _desc(FAR[name](), tmp_path)
    for t in range(d.c.n_types):
        assert d.c.tip_pair[t].kind == _abi.PAIR_LJ
        if not attraction:
            d.c.tip_pair[t].p[0] = 0.0
    scan = Scan(d, device=0)
    got, blocks = scan.grid_df()
    want = scan.grid()
    assert min(blocks) > 0
    size = np.linalg.norm(want[..., :3], axis=-1)
    assert (np.linalg.norm((got - want)[..., :3], axis=-1) / size).max() < 2.0 ** -38
    assert (np.abs(got - want)[..., 3] / np.abs(want[..., 3])).max() < 2.0 ** -38


def test_blocks_in_several_launches(tmp_path):
    """A grid of more blocks than are built at a time: the workspace stays below 67 MB
    of coefficients and a few of masks and tables, and the nodes are right on both
    sides of a launch's end."""
    torch = pytest.importorskip("torch")
    spec = small_slab(pixels=300, step=0.2, external=False)
    scan = Scan(_desc(spec, tmp_path), device=0)
    n, basis, origin = scan.grid_info()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _abi.check(_abi.lib().mafm_scan_build_grid(scan.handle, _abi.DF, None))
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] - 64 * np.prod(n) < 80e6
    got, blocks = scan.grid_df()
    assert np.prod(blocks) > 512
    # the same terms at every 400th node, the node wrapped into the cell as the build does
    spec.options["rigidgrid"] = "off"
    free_desc = _desc(spec, tmp_path)
    ijk = np.stack(np.unravel_index(np.arange(0, np.prod(n), 401), n), 1)
    pos = ijk * np.diag(basis) + origin
    cell, offset = np.array(free_desc.c.cell[:]).reshape(3, 3), np.array(free_desc.c.offset[:])
    turns = (pos - offset)[:, :2] / np.diag(cell)[:2]
    inside = (np.abs(turns - np.round(turns)) > 1e-9).all(1)   # either image is right on the border
    pos[:, :2] -= np.floor(turns) * np.diag(cell)[:2]
    want = Scan(free_desc, device=0).sample(pos[inside])
    have = got[tuple(ijk[inside].T)]
    size = np.linalg.norm(want[:, :3], axis=1)
    assert inside.mean() > 0.9
    assert (np.linalg.norm((have - want)[:, :3], axis=1) / size).max() < 1e-8   # positions of 30 A in other roundings
