"""The double-float relaxation's waiting for the warp's stage, which a lane leaves
out after heights of few steps: scans whose heights take one to a few steps, many,
and both in one warp take FP64's steps."""
import numpy as np
import pytest

from mechafm_gb300 import _abi, synth
from mechafm_gb300.scan import Input, Scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("opt", [dict(minterm="e", etol=1.0), dict(minterm="f", ftol=0.02), {}])
@pytest.mark.parametrize("integrator", ["midpoint", "rk4"])
def test_heights_of_few_and_many_steps(tmp_path, integrator, opt, lanes):
    spec = synth.cluster_60(n_atoms=24, area=2.0, step=0.1, zhigh=12.0, zlow=8.0, dz=0.4, integrator=integrator, **opt)
    scan = Scan(Input(spec.write(str(tmp_path))).desc(), device=0)
    want, _ = scan.run(_abi.FP64)
    got, _ = scan.run(_abi.DF, lanes=lanes)
    np.testing.assert_array_equal(got["steps"], want["steps"])
    np.testing.assert_allclose(got["tip"], want["tip"], rtol=0, atol=1e-8)
    np.testing.assert_allclose(got["force"], want["force"], rtol=1e-8, atol=1e-8)
