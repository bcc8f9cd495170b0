"""Neighbour pairs, pair histograms and observables from the cells of the last
rebuild, against all N^2 distances in float64 on the host: sizes around a
warp and a CTA, rows longer than the device orders, reflecting and periodic
boxes with few cells, and states in the middle of a rebuild period."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fluid(n, L, D, periodic, rs, seed, types=1):
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1.0 / D)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * D, indexing="ij"), -1).reshape(-1, D)
    g = g[rng.permutation(len(g))[:n]]
    x = (g + 0.5 + rng.uniform(-0.05, 0.05, g.shape)) * (L / side)
    r0 = min(0.6 * L / side, 0.8)  # no overlaps, whatever the density
    inter = [{"type": "lj", "pair": [a, b], "u0": 1.0, "r0": r0, "rc": 1.5 * r0, "n": 6}
             for a in range(types) for b in range(a, types) if (a, b) != (0, 1)]
    m = model.Model.from_dict({
        "n_dim": D, "l": np.full(D, L), "periodic": np.array(periodic, float), "dt": 1e-5,
        "n_steps": 10, "n_out": 1000, "tau_by_taud": np.ones(types), "seed": seed, "rs": rs,
        "interactions": inter, "reactions": []})
    t = rng.integers(0, types, n).astype(np.int32)
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    return model.SystemData(m, x, t, mol, np.arange(n, dtype=np.int32))


def _distances(x, L, periodic):
    d2 = np.zeros((len(x), len(x)))
    for k, per in enumerate(periodic):
        d = x[None, :, k] - x[:, None, k]
        if per > 0:
            d = d - L * np.round(d / L)
        d2 += d * d
    return np.sqrt(d2)


@pytest.mark.parametrize("n,L,D,periodic,rs,types", [
    (1, 9.0, 2, (1, 1), 2.0, 1), (33, 7.0, 2, (1, -1), 2.5, 1), (1037, 31.0, 2, (1, 1), 3.0, 2),
    (700, 20.0, 2, (-1, -1), 30.0, 1),   # every pair: rows beyond the ordered length
    (1201, 24.0, 2, (1, 1), 11.5, 2),    # long rows, stencil over the whole box
    (515, 9.0, 3, (1, 1, -1), 2.2, 2)])
def test_pairs_and_histogram_match_all_distances(n, L, D, periodic, rs, types):
    from pyrdsim_gb300.engine import Engine
    sd = _fluid(n, L, D, periodic, rs, seed=n, types=types)
    eng = Engine([sd])
    partners = np.ones((types, types), bool)
    if types > 1:
        partners[0, 1] = partners[1, 0] = False
    for steps in (0, 7, 6):  # the start, then the middle of two rebuild periods
        if steps:
            eng.step(steps)
        x, t = eng.state()
        r = _distances(x, L, periodic)
        i, j = np.nonzero(np.triu((r <= rs) & partners[t][:, t], 1))
        np.testing.assert_array_equal(eng.pairs(), np.stack([i, j], 1).astype(np.int32).reshape(-1, 2))
        r_max = 0.45 * L
        up = r[np.triu_indices(n, 1)]
        for bins in (1, 37, 5000):  # 5,000: float64 decides most bins
            width = r_max / bins
            want = np.bincount(np.minimum(np.floor(up[up < r_max] / width).astype(int), bins - 1),
                               minlength=bins)
            np.testing.assert_array_equal(eng.rdf_counts(r_max, bins), want)
    eng.close()


def test_pairs_after_a_failed_call():
    """A call that ends with a device error leaves particles anywhere: the
    pairs are still those of the current positions."""
    from pyrdsim_gb300.engine import Engine, EngineError
    sd = _fluid(300, 17.0, 2, (1, 1), 2.5, seed=4)
    eng = Engine([sd])
    xi = np.zeros((3, 300, 2))
    xi[:, ::7] = 300.0  # kicks far beyond the allowed displacement
    with pytest.raises(EngineError):
        eng.step(3, xi=xi, u1=np.ones((3, 300)), u2=np.ones((3, 300)))
    x, _ = eng.state()
    r = _distances(x, 17.0, (1, 1))
    i, j = np.nonzero(np.triu(r <= 2.5, 1))
    np.testing.assert_array_equal(eng.pairs(), np.stack([i, j], 1).astype(np.int32).reshape(-1, 2))
    eng.close()
