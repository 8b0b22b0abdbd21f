"""Two sessions of different materials side by side on one device: each works
with its own element matrix (smoothers, band groups, Galerkin operators,
sensitivities), so a session's results do not change by another one's set-up."""
import numpy as np
import pytest

from spgrid_topo_opt_b200 import configs, native

pytestmark = pytest.mark.gpu


def _results(prob, precision, other=None):
    """V-cycle, solve and sensitivities, before and after a density update;
    `other` is set up right after the session and solved in between."""
    out, inp = [], configs.to_inputs(prob)  # (a session updates its inputs' densities)
    with native.Session(inp, precision=precision) as s:
        second = native.Session(other, precision=precision) if other is not None else None
        rho = inp.density.data.copy()
        for scale in (1.0, 0.8):
            s.set_density(rho * scale)
            r = np.random.default_rng(2).standard_normal((3, len(s.flags(0)))) * ((s.flags(0) & 0x10) != 0)
            out.append(s.apply(native.OP_VCYCLE, 0, r))
            s.solve(tolerance=1e-6)
            out += [s.displacements(), *s.sensitivity()[1:], s.stencils(2)[0]]
            if second is not None:
                second.solve(tolerance=1e-6)
        if second is not None:
            second.close()
    return out


@pytest.mark.parametrize("precision", [native.PRECISION_REFERENCE, native.PRECISION_FP64, native.PRECISION_MIXED])
@pytest.mark.parametrize("n", [20, 64])  # band groups and short passes; also passes with a thread a node
def test_sessions_keep_their_material(native_lib, n, precision):
    prob = configs.cantilever_box(n, density=(0.2, 1.0), bottom_size=(n + 3) // 4)
    other = configs.to_inputs(prob, E=4e5, nu=0.45)
    for alone, beside in zip(_results(prob, precision), _results(prob, precision, other)):
        assert np.array_equal(alone, beside)
