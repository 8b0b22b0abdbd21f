"""The boundary-band groups of the V-cycle as cluster launches (band_group.cuh)
against the oracle's V-cycle: bands of a few hundred to several thousand nodes,
levels with and without stencils, and bands too large for a cluster's shared
memory, which run pass by pass.

FP64 V-cycles agree with the oracle to round-off (1e-10 of the field, as the
whole V-cycle in test_gpu_parity.py: sums of up to a few thousand terms in
another order, times the cycle's smoothing steps); the FP32 V-cycle of the
mixed mode to 1e-3 (FP32 rounding of 6e-8 times the condition of the bottom
level, up to 1e4 here).
"""
import numpy as np
import pytest

from oracle import oracle as orc
from spgrid_topo_opt_b200 import configs, native

pytestmark = pytest.mark.gpu


def _inputs(name):
    if name == "box9":        # 100 nodes a colour layer, CTAs with single nodes
        return configs.to_inputs(configs.cantilever_box(9, density=(0.2, 1.0), bottom_size=2))
    if name == "box33":       # odd faces
        return configs.to_inputs(configs.cantilever_box(33, density=(0.2, 1.0), bottom_size=4))
    if name == "shell40":     # ragged band, several stencil levels
        return configs.to_inputs(configs.sphere_shell(40, bottom_size=3))
    if name == "bridge":      # four separate bands
        return configs.to_inputs(configs.bridge(45, 13, 27, density=0.5, bottom_size=6, support_radius=0.08))
    return configs.to_inputs(configs.cantilever_box(72, density=(0.2, 1.0), bottom_size=8))  # box72: a large band


@pytest.mark.parametrize("name", ["box9", "box33", "shell40", "bridge", "box72"])
@pytest.mark.parametrize("precision,tol", [(native.PRECISION_FP64, 1e-10), (native.PRECISION_MIXED, 1e-3)])
def test_vcycle_with_band_groups(native_lib, name, precision, tol):
    inp = _inputs(name)
    o = orc.Oracle(inp, mode=orc.MODE_FP64)
    with native.Session(inp, precision=precision) as s:
        fl = s.flags(0)
        r = np.random.default_rng(5).standard_normal((3, len(fl))) * ((fl & 0x10) != 0)
        for v, bit in enumerate((0x20, 0x40, 0x80)):
            r[v][(fl & bit) != 0] = 0
        got, want = s.apply(native.OP_VCYCLE, 0, r), o.apply(orc.OP_VCYCLE, 0, r)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("name", ["box33", "shell40", "bridge"])
def test_reference_rounding_with_band_groups(native_lib, name):
    """Cast_To_Float after every band sweep inside a group: the oracle's
    iteration count, displacements to 1e-5 (test_gpu_parity.py's bounds)."""
    inp = _inputs(name)
    ref = orc.Oracle(inp, mode=orc.MODE_REF, tolerance=1e-6).solve()
    with native.Session(inp, precision=native.PRECISION_REFERENCE) as s:
        st = s.solve(tolerance=1e-6)
        d = s.displacements()
    assert st["iterations"] == ref["iterations"]
    want = ref["displacements"][..., :3]
    assert np.abs(d[..., :3] - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("precision", [native.PRECISION_FP64, native.PRECISION_MIXED])
def test_refused_band_is_examined_once(native_lib, precision):
    """The face of box80 is too large for a cluster on level 0, on level 2 (21^3
    nodes) its stencil rows are too large for a cluster's shared memory in FP64:
    density updates rebuild the operators and do not come back to it."""
    inp = configs.to_inputs(configs.cantilever_box(80, density=(0.2, 1.0), bottom_size=10))
    with native.Session(inp, precision=precision) as s:
        assert s.levels == 4
        for _ in range(2):
            s.set_density(inp.density.data)
        groups = [s.band_group(l) for l in range(s.levels)]
    assert groups[0] == (0, 1)
    assert (groups[2][0] > 0) == (precision == native.PRECISION_MIXED) and groups[2][1] == 1


@pytest.mark.parametrize("n,precision,level,on", [
    (48, native.PRECISION_MIXED, 0, True), (54, native.PRECISION_MIXED, 0, False),
    (54, native.PRECISION_FP64, 0, True), (56, native.PRECISION_FP64, 0, False),
    (82, native.PRECISION_MIXED, 2, True), (90, native.PRECISION_MIXED, 2, False),
    (68, native.PRECISION_FP64, 2, True)])
def test_lines_between_groups_and_passes(native_lib, n, precision, level, on):
    """band_slots(): faces just below and above the size from which the passes are
    faster launched one by one."""
    inp = configs.to_inputs(configs.cantilever_box(n, density=(0.2, 1.0), bottom_size=12))
    with native.Session(inp, precision=precision) as s:
        assert s.levels > level + 1
        assert (s.band_group(level)[0] > 0) == on


@pytest.mark.parametrize("precision", [native.PRECISION_REFERENCE, native.PRECISION_FP64, native.PRECISION_MIXED])
@pytest.mark.parametrize("name,on", [("box9", True), ("box33", True), ("shell40", True), ("bridge", True),
                                     ("box72", False)])
def test_which_inputs_run_level0_groups(native_lib, name, on, precision):
    """The inputs above that are meant to test the cluster launches run them on
    level 0, box72 the fallback."""
    with native.Session(_inputs(name), precision=precision) as s:
        assert (s.band_group(0)[0] > 0) == on
