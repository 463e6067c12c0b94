"""The surrogate's mma.sync pass with 8, 4, 2 lanes or one per particle (chosen
by the system's size) against its tcgen05 pass, on the same network."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POTENTIAL = "4*(r**-12-r**-6) + 0.5*exp(-(r-1.5)**2/0.02) + 0.1*cos(4*r)*exp(-r)"


def _sim(cells, dim):
    from dompap_gb300 import Simulation
    from dompap_gb300.positions import FCC, generate_positions

    unit = FCC if dim == 3 else ((0.0,) * 4,)
    pos = generate_positions(unit, cells, (1.0,) * dim)
    box = np.array(cells, dtype=np.float64)
    scale = (pos.shape[0] / np.prod(box) / 0.8) ** (1 / dim)
    box, pos = box * scale, pos * scale + np.random.default_rng(4).normal(0.0, 0.05, size=pos.shape)
    pos -= np.floor(pos / box) * box
    n = len(pos)
    sim = Simulation(positions=pos, velocities=np.zeros_like(pos), box_vectors=box, masses=np.ones(n),
                     particle_types=np.zeros(n, dtype=np.int32), neighbor_list_skin=0.3,
                     max_number_of_neighbors=512)
    sim.set_pair_potential(POTENTIAL, 3.0)
    sim.set_neighbor_list(skin=0.3, max_number_of_neighbors=512, method_str="cell list")
    return sim


@pytest.mark.parametrize("cells", [(5, 5, 5), (9, 9, 9), (14, 14, 13), (21, 20, 20), (27, 26, 26), (8, 8, 7, 7)],
                         ids=lambda c: "x".join(map(str, c)))
def test_lanes_per_particle(cells, monkeypatch):
    from dompap_gb300.mlp import PairSurrogate

    sur = PairSurrogate(POTENTIAL, 3.0, n_samples=4096, seed=1)
    out = {}
    for env in ("tcgen05", "mma"):
        monkeypatch.setenv("DOMPAP_MLP_TENSOR", env)
        sim = _sim(cells, len(cells))
        sim.set_pair_surrogate(sur)
        out[env] = (sim.get_forces(), sim.get_potential_energy(), sim.get_virial())
    (f, u, w), (g, v, x) = out["tcgen05"], out["mma"]
    # the same bf16 operands and float32 accumulation, summed in another order
    assert np.sqrt(np.mean((f - g) ** 2) / np.mean(f ** 2)) <= 1e-5
    assert abs(u - v) <= 1e-6 * abs(u) and abs(w - x) <= 1e-6 * np.sum(np.abs(f))
