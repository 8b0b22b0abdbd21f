"""The dense bottom inverse in nested-dissection order (bottom_order.hpp):
bottoms of several parts with padding between them, against the oracle's exact
bottom solve.  FP64, relative 1e-10 as test_bottom_solve_and_vcycle."""
import numpy as np
import pytest

from oracle import oracle as orc
from spgrid_topo_opt_b200 import configs, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["box44", "bridge72", "shell96"])
def test_bottom_solve_in_parts(native_lib, name):
    if name == "box44":        # 12^3 nodes: two halves and a plane
        inp = configs.to_inputs(configs.cantilever_box(44, density=(0.2, 1.0), bottom_size=16))
    elif name == "bridge72":   # 19 x 7 x 13 nodes, supports at four corners
        inp = configs.to_inputs(configs.bridge(72, 24, 48, density=0.5, bottom_size=20, support_radius=0.06))
    else:                      # a shell: parts with holes
        inp = configs.to_inputs(configs.sphere_shell(96, bottom_size=24))
    o = orc.Oracle(inp, mode=orc.MODE_FP64)
    with native.Session(inp, precision=native.PRECISION_FP64) as s:
        top = s.levels - 1
        fl = s.flags(top)
        b = np.random.default_rng(3).standard_normal((3, len(fl))) * ((fl & 0x10) != 0)
        got, want = s.apply(native.OP_BOTTOM, top, b), o.apply(orc.OP_BOTTOM, top, b)
        assert s.solve(tolerance=1e-2)["bottom_unknowns"] > 4096
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()


@pytest.mark.parametrize("precision,tol", [(native.PRECISION_FP64, 1e-9), (native.PRECISION_MIXED, 1e-4)])
def test_bottom_in_parts_after_a_density_update(native_lib, precision, tol):
    """New densities keep the order and its tables and fill the array again.  The
    right-hand side is nonzero on unknowns only, so the bound is relative to the
    solution: 1e-16 times the bottom's condition (stiffnesses of 0.008 to 1 over
    15 nodes across: up to 1e6) in FP64; in mixed precision the V-cycle applies
    an FP32 copy, whose rounding of 6e-8 grows by the cancellation in a row of
    10^4 random terms, up to 10^2 in each of the three phases."""
    prob = configs.cantilever_box(44, density=(0.2, 1.0), bottom_size=16)
    rho = prob.density.copy()
    prob.density = 1.2 - rho  # another design in the same range
    new = configs.to_inputs(prob)
    o = orc.Oracle(new, mode=orc.MODE_FP64)
    prob.density = rho
    with native.Session(configs.to_inputs(prob), precision=precision) as s:
        top = s.levels - 1
        fl, spokes = s.flags(top), s.stencils(top)[1]
        free = np.stack([((spokes & 0x07FFFFFF) != 0) & ((fl & bit) == 0) for bit in (0x20, 0x40, 0x80)])
        b = np.random.default_rng(4).standard_normal((3, len(fl))) * free
        before = s.apply(native.OP_BOTTOM, top, b)
        s.set_density(new.density.data)
        got, want = s.apply(native.OP_BOTTOM, top, b), o.apply(orc.OP_BOTTOM, top, b)
        assert s.solve(tolerance=1e-2)["bottom_unknowns"] > 4096
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
    assert np.abs(before - want).max() > 0.01 * np.abs(want).max()
