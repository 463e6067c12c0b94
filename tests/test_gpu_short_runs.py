"""Single steps of systems that run in groups of steps: one step kernel and no
idle ones, with the trajectory of a longer run bit for bit."""
import numpy as np
import pytest

from test_gpu_groups import _result, _system

pytestmark = pytest.mark.gpu


def test_a_step_is_two_launches(monkeypatch):
    from dompap_gb300 import _lib

    sim = _system(monkeypatch, True, 3, "fp32", False, 128)
    sim.run(3)
    for run in (sim.step, sim.step_leap_frog, lambda: sim.run(1)):
        run()
        assert int(_lib.load().dp_kernel_launches(sim._h)) == 2  # the step, the step counter


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dim,mixture", [(2, False), (3, True), (4, False)])
def test_single_steps_follow_a_run(monkeypatch, dim, mixture, precision):
    a, b, c = (_system(monkeypatch, True, dim, precision, mixture, 128) for _ in range(3))
    a.run(41)
    for _ in range(41):
        b.step()
    for steps in (1, 5, 1, 1, 12, 1, 20):
        c.run(steps)
    want = _result(a)
    assert want[4] >= 3  # rebuilds
    for sim in (b, c):
        for x, y in zip(want, _result(sim)):
            assert np.array_equal(x, y)


def test_far_positions_are_wrapped_by_a_single_step(monkeypatch):
    """The first step from positions outside the box (the reference's min-image
    path) leaves them wrapped, as a step in a group does."""
    a, b = (_system(monkeypatch, True, 3, "fp64", False, 128) for _ in range(2))
    box = np.array(a.box_vectors)
    for sim in (a, b):
        pos = np.array(sim.positions)
        pos[::7] += 2 * box
        pos[3::11] -= box
        sim.positions = pos
    a.run(2)
    b.run(1)
    b.run(1)
    for x, y in zip(_result(a), _result(b)):
        assert np.array_equal(x, y)
