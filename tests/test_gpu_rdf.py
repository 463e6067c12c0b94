"""The pair-distance histogram behind g(r) against np.histogram of the
oracle's distances, count for count: sizes at the edges of the kernel's tiles
(64 and 256 particles), every selection of types, uneven, degenerate and far
bin edges, and distances that sit exactly on an edge."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _counts(sim, edges, type_a=-1, type_b=-1):
    from dompap_gb300 import _lib

    sim._push()
    e = np.ascontiguousarray(edges, dtype=np.float64)
    out = np.zeros(e.size - 1, dtype=np.uint64)
    _lib.check(_lib.load().dp_rdf_counts(sim._h, type_a, type_b, _lib.dptr(e), e.size - 1,
                                         out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))))
    return out


def _expected(pos, box, edges, a, b):
    d = pos[a][:, None, :] - pos[b][None, :, :]
    for k in range(pos.shape[1]):
        d[:, :, k] -= box[k] * np.round(d[:, :, k] / box[k])
    q = d[:, :, 0] * d[:, :, 0]
    for k in range(1, pos.shape[1]):
        q = q + d[:, :, k] * d[:, :, k]
    return np.histogram(np.sqrt(q), bins=edges)[0].astype(np.uint64)


def _sim(pos, box, types):
    from dompap_gb300 import Simulation

    sim = Simulation(positions=pos, velocities=np.zeros_like(pos), box_vectors=box, particle_types=types,
                     masses=np.ones(len(pos)), neighbor_list_skin=0.1)
    return sim


EDGES = {
    "self": np.linspace(0.0, 4.0, 41),
    "one": np.array([0.0, 9.0]),
    "uneven": np.concatenate([[0.3, 0.30000001, 0.31], np.geomspace(0.5, 5.0, 37)]),
    "equal": np.array([0.2, 1.0, 1.0, 1.0, 2.0, 2.0, 3.5]),
    "below0": np.array([-2.0, -1.0, 0.0, 0.5, 4.0]),
    "beyond": np.array([1.0, 2.0, 50.0, np.inf]),
    "many": np.linspace(0.4, 4.4, 8193),
}


@pytest.mark.parametrize("n", [2, 63, 64, 65, 255, 257, 700])
@pytest.mark.parametrize("dim", [2, 3, 4])
def test_counts_equal_np_histogram(n, dim):
    rng = np.random.default_rng([n, dim])
    box = np.array([9.0, 8.5, 10.0, 9.5])[:dim]
    pos = rng.uniform(0.0, 1.0, size=(n, dim)) * box
    types = rng.integers(0, 3, size=n).astype(np.int32)
    sim = _sim(pos, box, types)
    everyone = np.arange(n)
    for name, edges in EDGES.items():
        for a, b in ((-1, -1), (0, 0), (0, 2), (2, 0), (-1, 1), (1, -1), (7, 7)):
            sel = [everyone if t < 0 else np.nonzero(types == t)[0] for t in (a, b)]
            got = _counts(sim, edges, a, b)
            assert np.array_equal(got, _expected(pos, box, edges, *sel)), (name, a, b)


@pytest.mark.parametrize("n", [1536, 1537, 1600])
@pytest.mark.parametrize("dim", [2, 3, 4])
def test_typed_counts_beside_the_line_between_the_two_forms(n, dim):
    """Up to 152 work items (256 particles x 64 partners; 1,536 particles have
    144, 1,537 have 175) the kernel compares the types, above they are selected."""
    rng = np.random.default_rng([n, dim, 1])
    box = np.array([9.0, 8.5, 10.0, 9.5])[:dim]
    pos = rng.uniform(0.0, 1.0, size=(n, dim)) * box
    types = rng.integers(0, 3, size=n).astype(np.int32)
    sim = _sim(pos, box, types)
    for a, b in ((-1, -1), (1, 1), (0, 2), (-1, 1), (1, -1), (7, 7)):
        sel = [np.arange(n) if t < 0 else np.nonzero(types == t)[0] for t in (a, b)]
        assert np.array_equal(_counts(sim, EDGES["uneven"], a, b), _expected(pos, box, EDGES["uneven"], *sel)), (a, b)


def test_distances_on_bin_edges():
    """A simple cubic lattice: every distance is the square root of an integer,
    and the edges are exactly those distances."""
    pos = np.stack(np.meshgrid(*[np.arange(8.0)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    box = np.array([8.0, 8.0, 8.0])
    sim = _sim(pos, box, np.zeros(len(pos), dtype=np.int32))
    edges = np.sqrt(np.arange(0.0, 20.0))
    everyone = np.arange(len(pos))
    assert np.array_equal(_counts(sim, edges), _expected(pos, box, edges, everyone, everyone))


def test_unwrapped_positions_and_a_moved_list():
    """Positions outside the box, and slots that a list build has reordered."""
    rng = np.random.default_rng(5)
    box = np.array([12.0, 12.5, 13.0])
    pos = rng.uniform(-1.5, 2.5, size=(900, 3)) * box
    types = rng.integers(0, 2, size=900).astype(np.int32)
    sim = _sim(pos, box, types)
    sim.set_neighbor_list(method_str="cell list")
    edges = np.linspace(0.1, 6.0, 60)
    one = np.nonzero(types == 1)[0]
    assert np.array_equal(_counts(sim, edges), _expected(pos, box, edges, np.arange(900), np.arange(900)))
    assert np.array_equal(_counts(sim, edges, 1, 1), _expected(pos, box, edges, one, one))
