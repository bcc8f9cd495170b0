"""Paths of the period kernel that only crowded places reach: chunks that touch
more particles than they stage, rows longer than the slot codes, rows beyond
the stored width.  States equal the per-step kernels' bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import _engine

pytestmark = pytest.mark.gpu

# particles, box, lanes per chain of the period kernel at that size
SIZES = [(6001, 60.0, 4), (20011, 110.0, 2), (40009, 155.0, 1)]


def _crowded(n, L, law, seed=1):
    """3,000 particles in one corner of the box (a few hundred neighbours each),
    ten clusters of 60, the others anywhere; three species that react."""
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, L, (n, 2))
    x[:3000] = rng.uniform(1.0, 7.0, (3000, 2))
    for q in range(10):
        x[3000 + 60 * q:3060 + 60 * q] = [L - 4.0, 4.0 + 5.0 * q] + rng.uniform(-0.4, 0.4, (60, 2))
    inter = [{"type": "tanh", "pair": [a, b], "u0": 0.02, "r0": 0.5, "a": 0.3, "rc": 1.0}
             for a in range(3) for b in range(a, 3)] if law else []
    m = model.Model.from_dict({
        "n_dim": 2, "l": np.array([L, L]), "periodic": np.array([1.0, 1.0]), "dt": 1e-4,
        "n_steps": 10, "n_out": 1000000, "tau_by_taud": np.ones(3), "seed": seed, "rs": 2.5,
        "interactions": inter,
        "reactions": [{"type": "locally_catalyzed", "reactant": 0, "product": 1, "catalyst": 1,
                       "rate": 5.0, "r0": 1.0},
                      {"type": "locally_inhibited", "reactant": 1, "product": 2, "rate": 60.0,
                       "rate_decrease": 0.5, "inhibitor": 0, "inhibitor2": 2, "r0": 1.0},
                      {"type": "linear", "reactant": 2, "product": 0, "rate": 30.0}]})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    return model.SystemData(m, x, rng.integers(0, 3, n).astype(np.int32), mol,
                            np.arange(n, dtype=np.int32))


def _same_as_per_step(sd, calls, **kw):
    """Steps the period kernel and the per-step kernels; returns the counts of
    the start's list and the number of type changes."""
    one, per_step = _engine([sd], **kw), _engine([sd], period_kernel=False, **kw)
    lists = one.test_lists()
    changed, prev = 0, one.state()[1]
    for k in calls:
        one.step(k)
        per_step.step(k)
        (xa, ta), (xb, tb) = one.state(), per_step.state()
        np.testing.assert_array_equal(ta, tb)
        np.testing.assert_array_equal(xa, xb)
        changed += int((ta != prev).sum())
        prev = ta
    np.testing.assert_array_equal(one.drift(), per_step.drift())
    one.close()
    per_step.close()
    return lists, changed


@pytest.mark.parametrize("n,L,lanes", SIZES)
def test_crowded_reactions_without_pair_laws(n, L, lanes):
    """Reactions that count neighbours in a system without pair laws: a chunk that
    stages nothing has no pair walk to hold it back, and must not run ahead of
    the particles it lists."""
    for _ in range(2):  # (the second run shows the same from run to run)
        lists, changed = _same_as_per_step(_crowded(n, L, law=False), (7, 64, 130, 99))
        assert lists["lanes"] == lanes and 0 < lists["unstaged"] < lists["chunks"], lists
        assert changed > 500, changed


@pytest.mark.parametrize("width,path", [(8, "beyond_width"), (200, "beyond_codes")])
@pytest.mark.parametrize("n,L,lanes", SIZES)
def test_long_rows_are_summed_in_list_order(n, L, lanes, width, path):
    """Rows that the codes or the stored width do not hold, with 1, 2 and 4 lanes per
    chain, in staged and unstaged chunks: the float32 sums in list order."""
    lists, changed = _same_as_per_step(_crowded(n, L, law=True), (5, 44, 31), list_width=width)
    assert lists["lanes"] == lanes and lists[path] > 0, lists
    assert 0 < lists["unstaged"] < lists["chunks"] and changed > 100, (lists, changed)


@pytest.mark.parametrize("n", [1009, 14593, 30011])
def test_rows_beyond_the_width_of_a_fluid(n):
    """The same in an even fluid, whose chunks are all staged."""
    from pyrdsim_gb300 import workloads
    sd = workloads.active_wall_fluid(n=n, seed=n, k_on=20.0, k_off=50.0)
    lists, _ = _same_as_per_step(sd, (3, 58, 24), list_width=8)
    assert lists["beyond_width"] > 100 and lists["unstaged"] == 0, lists


@pytest.mark.parametrize("n,D,rc,period", [(13824, 3, 2.5, 1), (35937, 3, 2.5, 1),
                                           (46656, 3, 2.5, 0), (60000, 2, 5.0, 1)])
def test_period_kernel_only_where_its_tables_hold_a_chunk(n, D, rc, period):
    """Large tables are cut to make every chunk resident; a system whose chunks would
    no longer fit them takes the per-step kernels."""
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(1)
    L = np.full(D, (n / 0.5) ** (1.0 / D))
    side = int(np.ceil(n ** (1.0 / D)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * D, indexing="ij"), -1).reshape(-1, D)[:n]
    x = (g + 0.5 + rng.uniform(-0.1, 0.1, (n, D))) * (L / side)
    m = model.Model.from_dict({
        "n_dim": D, "l": L, "periodic": np.ones(D), "dt": 1e-4, "n_steps": 10, "n_out": 1000000,
        "tau_by_taud": np.ones(1), "seed": 1,
        "interactions": [{"type": "yukawa", "pair": [0, 0], "u0": 10.0, "r0": 1.0, "rc": rc}]})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    sd = model.SystemData(m, x, np.zeros(n, np.int32), mol, np.arange(n, dtype=np.int32))
    e = _engine([sd])
    assert e.info()["period_kernel"] == period, e.test_lists()
    e.close()


@pytest.mark.parametrize("types", [3, 16])
@pytest.mark.parametrize("tpp", [1, 2, 4, 8])
@pytest.mark.parametrize("n,D", [(131, 1), (2177, 2), (1031, 3)])
def test_period_kernel_of_every_variant(n, D, tpp, types):
    """1 to 8 lanes per particle in 1D to 3D, up to the most species, reflecting and
    periodic edges, two laws on some pairs, reactions that count neighbours."""
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(n + types)
    side = int(np.ceil(n ** (1.0 / D)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * D, indexing="ij"), -1).reshape(-1, D)
    x = (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.1, 0.1, (n, D))) * 1.4
    pairs = [(a, b) for a in range(3) for b in range(a, 3)] + [(t, t) for t in range(3, types)]
    m = model.Model.from_dict({
        "n_dim": D, "l": np.full(D, 1.4 * side), "periodic": np.array([1.0] * (D - 1) + [-1.0]),
        "dt": 1e-4, "n_steps": 10, "n_out": 1000000, "tau_by_taud": np.ones(types), "seed": n,
        "rs": 3.6,
        "interactions": [{"type": "lj", "pair": [a, b], "u0": 1.0, "r0": 1.1, "rc": 2.5, "n": 6}
                         for a, b in pairs] +
                        [{"type": "yukawa", "pair": [0, 1], "u0": 3.0, "r0": 1.0, "rc": 2.2}],
        "reactions": [{"type": "linear", "reactant": 0, "product": types - 1, "rate": 30.0},
                      {"type": "locally_catalyzed", "reactant": types - 1, "catalyst": 1,
                       "product": 2, "rate": 5.0, "r0": 1.7},
                      {"type": "locally_inhibited", "reactant": 2, "product": 0, "rate": 60.0,
                       "rate_decrease": 2.0, "inhibitor": 1, "r0": 2.0}]})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    sd = model.SystemData(m, x, rng.integers(0, types, n).astype(np.int32), mol,
                          np.arange(n, dtype=np.int32))
    lists, changed = _same_as_per_step(sd, (6, 47, 30), threads_per_particle=tpp)
    assert lists["lanes"] == (4 if tpp == 2 and D < 3 else 1) and changed > 0, (lists, changed)


@pytest.mark.parametrize("n,rc", [(6000, 4.0), (8000, 4.0), (15000, 2.5), (16000, 2.5)])
def test_tables_hold_chunks_that_reach_over_a_row_of_cells(n, rc):
    """One lane per particle (chunks of 128) where a row of cells holds one or two
    chunks: each touches whole rows, which its table has room for."""
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(1)
    side = int(np.ceil(np.sqrt(n)))
    L = np.sqrt(n / 0.5)
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1)
    x = (g.reshape(-1, 2)[:n] + 0.5 + rng.uniform(-0.1, 0.1, (n, 2))) * (L / side)
    m = model.Model.from_dict({
        "n_dim": 2, "l": np.array([L, L]), "periodic": np.ones(2), "dt": 1e-5, "n_steps": 10,
        "n_out": 1000000, "tau_by_taud": np.ones(1), "seed": 1,
        "interactions": [{"type": "yukawa", "pair": [0, 0], "u0": 3.0, "r0": 1.0, "rc": rc}]})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    sd = model.SystemData(m, x, np.zeros(n, np.int32), mol, np.arange(n, dtype=np.int32))
    e = _engine([sd], threads_per_particle=1)
    lists = e.test_lists()
    assert lists["lanes"] == 1 and lists["unstaged"] == 0, lists
    e.close()
