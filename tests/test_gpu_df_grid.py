"""The double-float rigid grid's build with interpolated far terms, against the
FP64 build (every term at every node) through the relaxation over both: the
same steps on every point, tip and force within the 1e-8 of the golden
fixtures.  Sizes: blocks cut by the periodic wrap, a field on top, a molecule
with Morse and Coulomb terms inside the scan, grids whose axes do not divide
into blocks, and a sheared cell, where the direct build runs."""
import ctypes as C

import numpy as np
import pytest

from mechafm_gb300 import _abi, synth
from mechafm_gb300.scan import Input, Scan

pytestmark = pytest.mark.gpu


def small_slab(**kw):
    kw = {"zhigh": 18.0, "zlow": 17.85, **kw}
    return synth.slab(nlx=6, nly=6, layers=3, cell=(12.0, 12.0, 20.0), tip_charge=-0.02, **kw)


SPECS = {
    "wrap": lambda: small_slab(pixels=76, step=0.2, external=False),
    "wrap_ragged_field": lambda: small_slab(pixels=71, step=0.17, cube_n=(48, 48, 80)),
    "molecule": lambda: synth.cluster_60(n_atoms=600, area=7.9, step=0.2, zhigh=10.0, zlow=9.85, rigidgrid="on"),
    "one_height_of_blocks": lambda: synth.slab(pixels=17, zhigh=18.0, zlow=17.95, external=False),
    "sheared": lambda: small_slab(pixels=20, step=0.4, external=False, shear=0.2),
}


@pytest.mark.parametrize("name", SPECS)
def test_interpolated_build_matches_fp64(tmp_path, name):
    d = Input(SPECS[name]().write(str(tmp_path))).desc()
    scan = Scan(d, device=0)
    want, _ = scan.run(_abi.FP64)
    got, st = scan.run(_abi.DF)
    np.testing.assert_array_equal(got["steps"], want["steps"])
    np.testing.assert_allclose(got["tip"], want["tip"], rtol=0, atol=1e-8)
    np.testing.assert_allclose(got["force"], want["force"], rtol=1e-8, atol=1e-8)
    np.testing.assert_allclose(got["energy"], want["energy"], rtol=1e-8, atol=1e-8)


@pytest.mark.parametrize("lj,a", [(True, 1.5), (False, 1.5), (False, 3.0)])
def test_weak_forces_keep_their_relative_accuracy(tmp_path, lj, a):
    """The dummy 12 A above a slab of Morse and LJ or only Morse terms every force is small;
    relative to itself it stays within 1e-9 of FP64 (a term's rounding is about
    1e-13, a position's 1e-11 A times a)."""
    spec = small_slab(pixels=76, step=0.2, external=False, zhigh=26.0, zlow=25.85)
    spec.overwrites = [("O", t, "morse", 0.1, a, 3.2) for t in (("C",) if lj else ("C", "N"))]
    scan = Scan(Input(spec.write(str(tmp_path))).desc(), device=0)
    want, _ = scan.run(_abi.FP64)
    got, _ = scan.run(_abi.DF)
    np.testing.assert_array_equal(got["steps"], want["steps"])
    np.testing.assert_allclose(got["force"][:, 2], want["force"][:, 2], rtol=1e-9, atol=0)


def test_interpolated_rebuild_is_identical_and_can_be_captured(tmp_path):
    torch = pytest.importorskip("torch")
    d = Input(SPECS["wrap_ragged_field"]().write(str(tmp_path))).desc()
    scan = Scan(d, device=0)
    want, _ = scan.run(_abi.DF)
    L = _abi.lib()
    _abi.check(L.mafm_scan_build_grid(scan.handle, _abi.DF, None))
    np.testing.assert_array_equal(scan.run(_abi.DF)[0], want)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _abi.check(L.mafm_scan_build_grid(scan.handle, _abi.DF, C.c_void_p(stream.cuda_stream)))
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(scan.run(_abi.DF)[0], want)
