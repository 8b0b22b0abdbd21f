"""Soft material in the FP32 V-cycle: the determinant of a node's diagonal block
is the cube of its stiffness and leaves the FP32 range for stiffness scales of
about 1e-18 here (and on coarse levels, whose corner nodes carry a small share
of a soft cell, for ordinary ones).  diagonal_inverse scales the block first, so
the mixed solve is the FP64 solve's up to FP32 rounding of the preconditioner:
both stop at 1e-9 of the initial residual, displacements to 1e-6."""
import numpy as np
import pytest

from spgrid_topo_opt_b200 import configs, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("domain", ["box", "shell"])
def test_mixed_solve_of_soft_material(native_lib, domain):
    prob = (configs.cantilever_box(20, density=1e-6, bottom_size=4) if domain == "box"
            else configs.sphere_shell(40, bottom_size=4))
    prob.density = np.where(prob.density > 0, 1e-6, 0.0)
    inp = configs.to_inputs(prob, minimum_stiffness=1e-18)
    u, its = [], []
    for precision in (native.PRECISION_FP64, native.PRECISION_MIXED):
        with native.Session(inp, precision=precision) as s:
            its.append(s.solve(tolerance=1e-9)["iterations"])
            u.append(s.displacements()[..., :3])
    assert its[1] <= its[0] + 3
    assert np.abs(u[1] - u[0]).max() <= 1e-6 * np.abs(u[0]).max()
