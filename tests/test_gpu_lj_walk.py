"""The per-step drift kernel's Lennard-Jones walk in every instantiation (1, 2, 4
and 8 lanes per particle, 1D to 3D), whatever the size: drifts, states and types
equal the general walk's bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import _engine

pytestmark = pytest.mark.gpu


def _fluid(n, D, seed):
    """Two species on a jittered lattice, the pairs of each particle on both sides
    of the cutoff; some pairs are put exactly at it."""
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(seed)
    side = max(int(np.ceil(n ** (1.0 / D))), 4)
    a = 1.25
    g = np.stack(np.meshgrid(*[np.arange(side)] * D, indexing="ij"), -1).reshape(-1, D)
    x = (g[rng.permutation(len(g))[:n]] + 0.5) * a
    x[n // 2:] += rng.uniform(-0.1, 0.1, x[n // 2:].shape)  # (the others: distances equal)
    m = model.Model.from_dict({
        "n_dim": D, "l": np.full(D, side * a), "periodic": np.ones(D), "dt": 1e-5,
        "n_steps": 10, "n_out": 1000000, "tau_by_taud": np.ones(2), "seed": seed, "rs": 3.2,
        "interactions": [{"type": "lj", "pair": [p, q], "u0": 1.0, "r0": 1.0, "rc": 2 * a, "n": 6}
                         for p, q in ((0, 0), (0, 1), (1, 1))],
        "reactions": [{"type": "linear", "reactant": 0, "product": 1, "rate": 100.0}]})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    return model.SystemData(m, x, rng.integers(0, 2, n).astype(np.int32), mol,
                            np.arange(n, dtype=np.int32))


@pytest.mark.parametrize("width", [0, 8])  # (8: rows beyond the stored width)
@pytest.mark.parametrize("tpp", [1, 2, 4, 8])
@pytest.mark.parametrize("n,D", [(1, 2), (65, 1), (2049, 2), (1031, 3)])
def test_lj_walk_of_every_variant(n, D, tpp, width):
    sd = _fluid(n, D, seed=n)
    walk, general = (_engine([sd], period_kernel=False, threads_per_particle=tpp,
                             list_width=width) for _ in range(2))
    walk.test_lj_walk(1)
    general.test_lj_walk(-1)
    if width and n > 65:
        assert walk.test_lists()["beyond_width"] > 0
    x, t = walk.state()
    for e in (walk, general):
        e.set_state(x, t)  # the start's drift by the chosen walk
    np.testing.assert_array_equal(walk.drift(), general.drift())
    for k in (1, 30):
        for e in (walk, general):
            e.step(k)
        for p, q in zip(walk.state(), general.state()):
            np.testing.assert_array_equal(p, q)
        np.testing.assert_array_equal(walk.drift(), general.drift())
    walk.close()
    general.close()
