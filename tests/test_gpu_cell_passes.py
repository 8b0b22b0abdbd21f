"""Level-0 colour passes on both sides of the lines between eight threads and one
thread per node (GS_CELL_NODES: nodes a pass, by precision and layout), against
the oracle.  Boxes of n^3 cells have about (n + 1)^3 / 8 nodes a pass.  Bounds
as in test_gpu_parity.py: FP64 sweeps 1e-11, V-cycles 1e-10; FP32 V-cycles 1e-3
as in test_gpu_band_groups.py."""
import numpy as np
import pytest

from oracle import oracle as orc
from spgrid_topo_opt_b200 import configs, native

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def _field(s, rng):
    fl = s.flags(0)
    f = rng.standard_normal((3, len(fl))) * ((fl & 0x10) != 0)
    for v, bit in enumerate((0x20, 0x40, 0x80)):
        f[v][(fl & bit) != 0] = 0
    return f


@pytest.mark.parametrize("n", [66, 72])
def test_planar_sweeps(native_lib, n):
    inp = configs.to_inputs(configs.cantilever_box(n, density=(0.2, 1.0), bottom_size=(n + 3) // 4))
    o = orc.Oracle(inp, mode=orc.MODE_FP64)
    rng = np.random.default_rng(n)
    with native.Session(inp, precision=native.PRECISION_REFERENCE) as s:
        u, b = _field(s, rng), _field(s, rng)
        for arg in (1, 2):  # full forward, boundary band backward
            assert _rel(s.apply(native.OP_SMOOTH, 0, u, b, arg=arg), o.apply(orc.OP_SMOOTH, 0, u, b, arg=arg)) < 1e-11


@pytest.mark.parametrize("n,precision,tol", [(25, native.PRECISION_FP64, 1e-10), (28, native.PRECISION_FP64, 1e-10),
                                             (50, native.PRECISION_MIXED, 1e-3), (56, native.PRECISION_MIXED, 1e-3)])
def test_packed_passes_in_the_vcycle(native_lib, n, precision, tol):
    inp = configs.to_inputs(configs.cantilever_box(n, density=(0.2, 1.0), bottom_size=(n + 3) // 4))
    o = orc.Oracle(inp, mode=orc.MODE_FP64)
    with native.Session(inp, precision=precision) as s:
        r = _field(s, np.random.default_rng(n))
        assert _rel(s.apply(native.OP_VCYCLE, 0, r), o.apply(orc.OP_VCYCLE, 0, r)) <= tol
