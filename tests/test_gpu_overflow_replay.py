"""A region that outgrows its room in the middle of a run: the steps after that
build ran on empty lists, so nothing they produced counts - not even a force
that became infinite. The steps are done again with more room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE, PER_AXIS, DT, FOCUS, SPEED = 15.46, 3, 0.001, 45, 12.0


def _system(precision):
    """27 swarms of particles without forces (epsilon 0), each collapsing to a
    point after FOCUS steps and apart again: in between, the regions around the
    27 points hold three times what the mean density suggests. Around each
    point nine pairs of interacting particles approach head-on; without forces
    the two would coincide exactly after 82 to 104 steps."""
    from dompap_gb300 import Simulation

    rng = np.random.default_rng(31)
    box = np.full(3, SIDE * PER_AXIS)
    centres = (np.stack(np.meshgrid(*[np.arange(PER_AXIS)] * 3, indexing="ij"), axis=-1).reshape(-1, 3) + 0.5) * SIDE
    centres = centres + rng.uniform(-0.3, 0.3, size=centres.shape)
    grid = (np.stack(np.meshgrid(*[np.arange(11)] * 3, indexing="ij"), axis=-1).reshape(-1, 3) + 0.5) / 11 - 0.5
    pos, vel, types = [], [], []
    meet = 82
    for c in centres:
        x = grid * SIDE + rng.normal(0.0, 0.2, size=grid.shape)
        to = rng.normal(0.0, 0.5, size=grid.shape)
        pos.append(c + x)
        vel.append((to - x) / (FOCUS * DT))
        types.append(np.ones(len(x)))
        for y in (-1.6, 0.0, 1.6):
            for z in (-1.6, 0.0, 1.6):
                half = np.array([meet * SPEED * DT, 0.0, 0.0])
                pos.append(c + [0.0, y, z] + np.array([-half, half]))
                vel.append(np.array([[SPEED, 0.0, 0.0], [-SPEED, 0.0, 0.0]]))
                types.append(np.zeros(2))
                meet = 82 + (meet - 82 + 7) % 23
    pos, vel = np.concatenate(pos), np.concatenate(vel)
    types = np.concatenate(types).astype(np.int32)
    pos = pos - np.floor(pos / box) * box
    np.random.seed(3)
    sim = Simulation(positions=pos, velocities=vel, box_vectors=box, masses=np.ones(len(pos)), particle_types=types,
                     neighbor_list_skin=1.4, max_number_of_neighbors=2048, precision=precision)
    sim.set_pair_potential("r**-6", 1.4)
    sim.set_pair_potential_parameters(sigma=np.ones((2, 2)), epsilon=np.array([[1.0, 0.0], [0.0, 0.0]]))
    sim.set_neighbor_list(skin=1.4, max_number_of_neighbors=2048, method_str="cell list")
    sim.set_integrator(time_step=DT)
    assert len(pos) / np.prod(box) * 4 / 3 * np.pi * 2.8**3 >= 32.0  # float32: on bricks
    return sim, types


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_steps_after_an_overflow_do_not_count(precision):
    steps = 110
    a, types = _system(precision)
    a.run_leap_frog(steps)
    # the same steps one at a time: every build is checked before a step uses it
    b, _ = _system(precision)
    for _ in range(steps):
        b.step_leap_frog()
    for name, bound in (("positions", 1e-6), ("velocities", 1e-3)):
        # same lists and forces: at most the order of equal sums differs
        # (6e-8 of forces up to ~2,000 for ~20 steps of 0.001)
        assert np.max(np.abs(np.array(getattr(a, name)) - np.array(getattr(b, name)))) <= bound
    # the pairs bounced: every one of the two turned back
    assert np.all(np.abs(np.array(a.velocities)[types == 0, 0]) > 1.0)
