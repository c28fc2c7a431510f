"""The two forms of the time step, a block per slice (small beams) and a warp per
slice (step_kernel, above 6 slices per SM), beyond what the small beams of the other
tests reach."""
import numpy as np
import pytest

import bb_pd_b200 as bb
from test_gpu_solver import LAWKW, compare, orun

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(24, 5, 6), (60, 9, 13), (31, 30, 31)])
@pytest.mark.parametrize("law,scheme", [("trilinear", "adr"), ("linear", "eulercromer"), ("exponential", "eulercromer")])
def test_coordinates_leave_the_fast_range_within_a_launch(nx, ny, nz, law, scheme):
    """The loaded nodes lie at z = 0 and move by less than 2^-100 in the first step,
    where the division by shared reciprocals no longer holds: the launch goes over to
    IEEE operations from its second step on. Lengths off by up to 4 s0 keep the laws busy."""
    inp = dict(bb.beam.build(bb.beam.small(nx=nx, ny=ny, nz=nz)))
    X = inp["undeformedCoordinates"].copy(order="F")
    X[:, 2] -= X[:, 2].max()
    rng = np.random.default_rng(nx)
    inp["undeformedCoordinates"] = X
    inp["UNDEFORMEDLENGTH"] = inp["UNDEFORMEDLENGTH"] * (1 + 1e-4 * rng.integers(-4, 5, inp["nBonds"]))
    kw = dict(LAWKW[law], scheme=scheme, amplitude="smoothstep", applied_final=-1e-4, n_time_steps=2_000_000_000)
    s = bb.Solver(inp, **kw)
    r = orun(inp, **kw)
    s.step(12)
    r.step(1)
    z = r.get("deformed")[X[:, 2] == 0, 2]
    assert ((z != 0) & (np.abs(z) < 2.0 ** -100)).any()
    r.step(11)
    compare(s, r, law)
    s.step(3)
    r.step(3)
    compare(s, r, law)
    s.close()
