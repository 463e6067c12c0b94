"""Float32 systems with a costly generated potential: they run on lists of slots
(two passes, the pair terms for kept entries only), cheap ones on bricks; the
choice follows the calls in the generated force, and a costly step costs no more
than its pair terms do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LJ = "4*(r**-12-r**-6)"
COSTLY = LJ + "".join(f" + 0.05*exp(-(r-{1.0 + 0.2 * k})**2/0.05)*cos({3 + k}*r)" for k in range(8))
CHEAP = [LJ, "(1-r/3)**2", "r**-12 + exp(-r)/r", "(1-exp(-2*(r-1.1)))**2", "1000*exp(-6*r) - r**-6", "r**-9.5",
         "r**-12 + tanh(3*(r-1.5))", "Harmonic repulsive"]
DEAR = [COSTLY, LJ + " + 0.1*cos(4*r)*exp(-r)", "r**-9.5 - 0.5*r**-4.2"]


def _sim(potential, cells, r_cut=3.0):
    from dompap_gb300 import Simulation
    from dompap_gb300.positions import FCC, generate_positions

    pos = generate_positions(FCC, cells, (1.0,) * 3)
    scale = (4 / 0.8) ** (1 / 3)
    box, pos = np.array(cells, dtype=np.float64) * scale, pos * scale
    rng = np.random.default_rng(2)
    pos = pos + rng.normal(0.0, 0.05, size=pos.shape)
    pos -= np.floor(pos / box) * box
    np.random.seed(4)
    sim = Simulation(positions=pos, velocities=rng.normal(size=pos.shape), box_vectors=box, masses=np.ones(len(pos)),
                     particle_types=np.zeros(len(pos), dtype=np.int32), neighbor_list_skin=0.3,
                     max_number_of_neighbors=256, precision="fp32")
    sim.set_pair_potential(potential, r_cut)
    sim.set_neighbor_list(skin=0.3, max_number_of_neighbors=256, method_str="cell list")
    sim.set_integrator(time_step=0.004, target_temperature=1.0, temperature_damping_time=0.1)
    return sim


@pytest.mark.parametrize("potential", CHEAP + DEAR)
def test_which_lists(potential):
    sim = _sim(potential, (14, 14, 14))
    if potential == "Harmonic repulsive":  # its cut is 1: too few neighbours for bricks
        sim.set_neighbor_list(skin=2.0, max_number_of_neighbors=256, method_str="cell list")
    sim.update_neighbor_list(check=False)
    # 4 lanes a particle either way; bricks are compiled for 4 CTAs an SM, slots for
    # 6, or 4 where the pair terms need the registers
    assert sim.get_step_launch() == ((4, 6) if potential in DEAR[1:] else (4, 4))


def test_costly_step_time():
    """108,000 particles: the costly force is eight times two calls of ~30
    instructions and an exp over Lennard-Jones' ~15, for a third of the listed
    pairs of a step that also walks them and integrates: about five Lennard-Jones
    steps (13 where every listed entry paid for it)."""
    ms = {}
    for name, potential in (("lj", LJ), ("costly", COSTLY)):
        sim = _sim(potential, (30, 30, 30))
        sim.run(10)
        ms[name] = min(sim.run_timed(40) for _ in range(3))
    assert ms["costly"] <= 7.0 * ms["lj"]


def test_costly_replicas_time():
    """256 replicas of 2,048: the costly force a dozen times Lennard-Jones' at most
    (8 here; more than 30 where it was inlined into every entry of the loop)."""
    from dompap_gb300.batched import Replicas, ReplicaSpec
    from dompap_gb300.positions import FCC, generate_positions

    scale = (4 / 0.8) ** (1 / 3)
    pos, box = generate_positions(FCC, (8, 8, 8), (1.0,) * 3) * scale, np.full(3, 8 * scale)
    rng = np.random.default_rng(3)
    specs = []
    for _ in range(256):
        p = pos + rng.normal(0.0, 0.05, size=pos.shape)
        specs.append(ReplicaSpec(p - np.floor(p / box) * box, rng.normal(size=p.shape), box, 1.0))
    ms = {}
    for name, potential in (("lj", LJ), ("costly", COSTLY)):
        replicas = Replicas(specs, potential, 3.0, seed=1)
        replicas.run(3)
        ms[name] = min(replicas.run(20) for _ in range(3))
    assert ms["costly"] <= 12.0 * ms["lj"]


@pytest.mark.parametrize("cells", [(5, 5, 5), (14, 14, 14)])
def test_forces_agree_with_float64(cells):
    a = _sim(COSTLY, cells)
    f = a.get_forces()
    u, w = a.get_potential_energy(), a.get_virial()
    a.set_precision("fp64")
    g = a.get_forces()
    # float32 terms: a few roundings (6e-8) of terms up to ~20 times the sum
    assert np.sqrt(np.mean((f - g) ** 2) / np.mean(g**2)) <= 5e-6
    assert abs(u - a.get_potential_energy()) <= 5e-6 * abs(a.get_potential_energy())
    assert abs(w - a.get_virial()) <= 2e-5 * np.sum(np.abs(g)) / 3
