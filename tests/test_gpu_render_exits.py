"""Rays that leave the volume end there (render.cu): against the oracle's rays,
which always take all their steps.  Axis-parallel and mirrored rays, an eye
inside the volume, empty space a negative threshold lets through, a slice.  The
images agree as in test_render.py: CUDA's and numpy's cos, sin and exp differ in
the last bits."""
import numpy as np
import pytest

from oracle import render_oracle as ro
from spgrid_topo_opt_b200 import configs, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,view,kw", [
    (0, (0, 0, 0, 0, 0, -5), dict(threshold=0.3)),
    (0, (-20, 30, 0, 0, 0, -5), dict(threshold=0.0)),
    (0, (15, -40, 0, 0, 0, -5), dict(threshold=-0.5)),
    (0, (10, 25, 5, 0, 0, -0.2), dict(threshold=0.6, mirror="xy")),
    (1, (0, 0, 0, 0, 0, -0.1), dict(threshold=0.01, extinction=2.0)),
    (1, (35, 60, 0, 0, 0, -4), dict(threshold=0.02, extinction=3.0, mirror="z", slice_=0.6)),
])
def test_early_exits(native_lib, mode, view, kw):
    prob = configs.cantilever_box(20, density=(0.05, 1.0), bottom_size=4)
    prob.density[4:16, 8:20, :] = 0.0
    inp = configs.to_inputs(prob)
    cam = native.view_matrix(*view)
    got, res = native.render(inp.density.base, inp.density.data, 64, 48, cam, mode=mode, frames=2, seed=3, **kw)
    ref, rres = ro.render(inp.density.base, inp.density.data, 64, 48, cam, mode=mode, frames=2, seed=3, **kw)
    assert res.tolist() == list(rres)
    ch = [(got >> s) & 0xFF for s in (0, 8, 16)], [(ref >> s) & 0xFF for s in (0, 8, 16)]
    diff = np.max([np.abs(a.astype(int) - b.astype(int)) for a, b in zip(*ch)], axis=0)
    assert np.mean(diff == 0) >= 0.995 and np.mean(diff <= 1) >= 0.999
