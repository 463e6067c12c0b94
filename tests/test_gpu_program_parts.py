"""A program holds the kernels that its system's size uses: every sum and every launch
shape works at sizes of each kind, and agrees with float64 on the whole."""
import numpy as np
import pytest

from test_gpu_bricks import _lattice, _sim

pytestmark = pytest.mark.gpu


# up to 8,192 (a warp a particle), up to 65,536 (four lanes), above
@pytest.mark.parametrize("counts", [(20, 20, 20), (21, 20, 20), (40, 40, 40), (41, 41, 40)], ids=str)
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("mixture", [False, True])
def test_every_kernel_of_a_size(counts, precision, mixture):
    pos, box = _lattice(counts, 1.06, np.random.default_rng(7), 0.05)
    types = (np.arange(len(pos)) % 2).astype(np.int32) if mixture else None
    sim = _sim(pos, box, 2.5, 0.3, precision, capacity=192, types=types)
    f, u, w, lap = sim.get_forces(), sim.get_potential_energy(), sim.get_virial(), sim.get_laplacian()
    assert np.all(np.isfinite(f)) and np.all(np.isfinite(lap)) and np.isfinite(u) and np.isfinite(w)
    # Newton's third law: the forces add up to roundings of a few of them
    assert np.max(np.abs(np.sum(f, axis=0))) <= (1e-5 if precision == "fp32" else 1e-11) * np.sum(np.abs(f))
    sim.set_integrator(time_step=0.002, target_temperature=1.0, temperature_damping_time=0.1)
    start = np.array(sim.positions), np.array(sim.velocities)
    ends = []
    for lanes in (0, 1, 4, 32):
        sim.positions, sim.velocities = start
        sim.set_step_launch(lanes, 0)
        sim.run_leap_frog(4)
        ends.append(np.array(sim.positions))
    for e in ends[1:]:
        d = e - ends[0]
        # float32 sums in another order: 6e-8 of forces up to ~300, 4 steps of 0.002
        assert np.max(np.abs(d - box * np.round(d / box))) <= 1e-7
