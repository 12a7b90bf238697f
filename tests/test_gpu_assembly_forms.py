"""The adjoint assembly of viscous 2D blocks with and without the diffusion: the
same numbers, on the tiles that were set or tuned."""
import math

import numpy as np
import pytest

from magudi_gb300 import capi, configs
from magudi_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def problem(n, ny, curvilinear=False, **kw):
    P = configs.monopole_2d(n=n, ny=ny, n_steps=6, save_interval=2, half_width=7.0, dt=0.02, target_center=(0.0, 3.0),
                            **kw)
    if curvilinear:
        P.options.curvilinear = True
        x, y = P.blocks[0].coordinates
        k = math.pi / 7.0
        P.blocks[0].coordinates = np.ascontiguousarray(np.stack(
            [x + 0.28 * np.sin(k * x) * np.sin(k * y), y + 0.28 * np.sin(k * y) * np.sin(0.5 * k * x)]))
    return P


def gradient(s, P, resident):
    s.set_trajectory_storage(resident)
    s.set_field(1, capi.FIELD_CONSERVED, P.blocks[0].initial_state)
    J = s.run_forward(P.n_steps, P.save_interval)
    return J, s.run_adjoint(), s.gradient(4 * P.n_steps), s.get_field(1, capi.FIELD_ADJOINT)


def same(a, b):
    return a[:2] == b[:2] and np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])


@pytest.mark.parametrize("curvilinear", [False, True])
@pytest.mark.parametrize("composite", [True, False])
def test_forms_are_bitwise_equal(curvilinear, composite):
    """Resident runs of 25,000 points form the diffusion in the assembly,
    checkpointed ones beside the recomputation do not."""
    P = problem(201, 127, curvilinear, composite_dissipation=composite)
    s = Solver(P)
    checkpointed = gradient(s, P, False)
    assert s.assembly_launch()[0] == 0
    resident = gradient(s, P, True)
    assert s.assembly_launch()[0] == 1
    assert same(checkpointed, resident)


def test_a_tile_that_was_set_is_the_one_launched():
    P = problem(201, 127)
    s = Solver(P)
    want = gradient(s, P, False)
    for tile in [(8, 8, 1), (4, 8, 1), (16, 8, 1)]:
        assert s.stage_tile(5, tile) == tile
        for resident in (False, True):
            assert same(gradient(s, P, resident), want)
            assert s.assembly_launch() == (int(resident), tile)
            assert s.stage_tile(5) == tile


def test_setup_tunes_the_form_with_the_diffusion():
    """Between the two lines on the number of points both forms run, and both are
    tuned: at 201x201 compact tiles of 64 points are 10% ahead of the tile before
    tuning."""
    assert Solver(problem(201, 201)).stage_tile(5) != (32, 4, 1)


def test_run_level_tuning_keeps_a_tile_it_timed():
    """The tile that checkpointed tuning runs leave is that of the kernel they
    launched, and the other form's stays as it was."""
    P = problem(201, 129)
    s = Solver(P)
    with_diffusion = s.stage_tile(5)
    s.tune_run(4, 2)
    tuned = s.stage_tile(5)
    gradient(s, P, False)
    assert s.assembly_launch() == (0, tuned)
    gradient(s, P, True)
    assert s.assembly_launch() == (1, with_diffusion)


def test_kernels_that_no_run_launches_are_not_tuned():
    P = problem(43, 39)
    s = Solver(P)
    assert s.assembly_launch() is None
    assert s.stage_tile(4) == (32, 4, 1)  # the tile before tuning
    s.tune_run(4, 2)
    assert s.stage_tile(4) == (32, 4, 1)
