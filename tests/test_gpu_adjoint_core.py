"""The adjoint RHS of random states on the smallest far-field boxes against
the oracle: every point next to faces, edges and corners (up to three
far-field entries a point), Cartesian and curvilinear, in 2D and 3D."""
import numpy as np
import pytest

import oracle_lib
from helpers import rel_err
from magudi_gb300 import capi, configs
from magudi_gb300.problem import Block, Options, Patch, Problem, quiescent_state
from magudi_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def far_field_box(sizes, curvilinear, viscous):
    nD = len(sizes)
    axes = np.meshgrid(*[np.linspace(0.0, 1.0 + 0.2 * d, n) for d, n in enumerate(reversed(sizes))], indexing="ij")
    x = [a.ravel() for a in reversed(axes)]
    if curvilinear:
        s = np.prod([np.sin(2.0 * c) for c in x], axis=0)
        x = [c + 0.02 * (d + 1) * s for d, c in enumerate(x)]
    N = int(np.prod(sizes))
    opts = Options(n_dimensions=nD, viscous=viscous, dissipation=True, dissipation_amount=0.01, curvilinear=curvilinear,
                   use_constant_cfl=False, time_step_size=1e-3, reynolds_number=100.0)
    block = Block(grid_size=tuple(sizes) + (1,) * (3 - nD), coordinates=np.ascontiguousarray(np.stack(x)),
                  initial_state=quiescent_state(N, nD, 1.4), target_state=quiescent_state(N, nD, 1.4))
    patches = []
    for d in range(nD):
        for end in (1, -1):
            e = [1, -1, 1, -1, 1, -1]
            e[2 * d], e[2 * d + 1] = end, end
            patches.append(Patch(f"farField.{d}.{end}", "SAT_FAR_FIELD", 1, end * (d + 1), tuple(e)))
    return Problem(options=opts, blocks=[block], patches=patches)


@pytest.mark.parametrize("sizes", [(25, 26), (33, 25), (25, 25, 25)])
@pytest.mark.parametrize("curvilinear", [False, True])
@pytest.mark.parametrize("viscous", [True, False])
@pytest.mark.parametrize("lanes", [1, 2])
def test_adjoint_rhs_on_far_field_boxes(sizes, curvilinear, viscous, lanes):
    if lanes == 2 and len(sizes) == 3:
        pytest.skip("two threads per point only in 2D")
    P = far_field_box(sizes, curvilinear, viscous)
    rng = np.random.default_rng(5)
    q = configs.random_state(P.blocks[0].n_points, len(sizes), 1.4, rng)
    lam = rng.uniform(-1.0, 1.0, q.shape)
    g, o = Solver(P), oracle_lib.Oracle(P)
    assert g.adjoint_core_lanes(lanes) == lanes
    for s in (g, o):
        s.set_field(1, capi.FIELD_CONSERVED, q)
        s.set_field(1, capi.FIELD_ADJOINT, lam)
        s.update_state()
        s.compute_rhs(capi.ADJOINT, 0.0, 0.0)
    assert rel_err(g.get_field(1, capi.FIELD_RHS), o.get_field(1, capi.FIELD_RHS)) < 1e-12
