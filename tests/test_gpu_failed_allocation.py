"""An allocation that the GPU cannot give is an error of that call, and the handle
stays usable: no buffer is taken for as large as it was asked to be."""
import numpy as np
import pytest

from test_gpu_bricks import _lattice, _sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(12, 12, 12), (23, 22, 21)], ids=str)  # rows; cell lists
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_lists_too_long_to_allocate(counts, precision):
    from dompap_gb300._lib import DompapGPUError

    pos, box = _lattice(counts, 1.06, np.random.default_rng(1), 0.05)
    sim, other = (_sim(pos, box, 2.5, 0.3, precision, capacity=192) for _ in range(2))
    before = sim.get_forces()
    for call in (lambda: sim.set_neighbor_list(skin=0.3, max_number_of_neighbors=2**30, method_str="cell list"),  # 4 GB a particle
                 sim.get_forces, lambda: sim.run_leap_frog(3), sim.get_potential_energy):
        with pytest.raises(DompapGPUError, match="cudaMalloc"):
            call()
    sim.set_neighbor_list(skin=0.3, max_number_of_neighbors=192, method_str="cell list")
    assert np.array_equal(sim.get_forces(), before)
    for s in (sim, other):
        s.set_integrator(time_step=0.004)
        s.run_leap_frog(30)
    assert np.max(np.abs(np.array(sim.positions) - np.array(other.positions))) <= 1e-4
