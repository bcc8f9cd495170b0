"""The float64 drift kernel at the sizes where its split changes (2, 4 and 16
particles per warp), ragged last chunks and rows beyond the stored width, in
2D and 3D, against the CPU oracle and against itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, D, law):
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1.0 / D)))
    L = max(side * 1.4, 8.0)
    g = np.stack(np.meshgrid(*[np.arange(side)] * D, indexing="ij"), -1).reshape(-1, D)
    x = (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.1, 0.1, (n, D))) * (L / side)
    inter = {"lj": {"type": "lj", "u0": 1.0, "r0": 1.1, "rc": 2.5, "n": 6},
             "lj5": {"type": "lj", "u0": 1.0, "r0": 1.1, "rc": 2.0, "n": 5},
             "yukawa": {"type": "yukawa", "u0": 3.0, "r0": 1.0, "rc": 2.5}}[law]
    m = model.Model.from_dict({
        "n_dim": D, "l": np.full(D, L), "periodic": np.ones(D), "dt": 1e-5, "n_steps": 10,
        "n_out": 1000, "tau_by_taud": np.array([1.0]), "seed": 1,
        "interactions": [dict(inter, pair=[0, 0])], "reactions": []})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    return model.SystemData(m, x, np.zeros(n, np.int32), mol, np.arange(n, dtype=np.int32))


@pytest.mark.parametrize("n,D,law", [(1, 2, "lj"), (9, 2, "lj5"), (1037, 2, "yukawa"),
                                     (6007, 2, "lj"), (40009, 2, "lj"), (2200, 3, "lj")])
def test_float64_drift_at_every_split(n, D, law):
    from oracle.oracle import Oracle
    from pyrdsim_gb300.engine import Engine
    sd = _system(n, D, law)
    ref = Oracle(sd, history_quirk=False).drift()
    floor = max(np.sqrt((ref ** 2).sum(1).mean()), 1e-300)
    first = None
    for tpp, width in ((2, 0), (2, 8), (1, 0), (8, 0)):
        eng = Engine([sd], precision="float64", threads_per_particle=tpp, list_width=width)
        a = eng.drift()
        err = np.linalg.norm(a - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), floor)
        assert err.max() < 1e-12, (tpp, width, err.max())
        if tpp == 2:  # the sums do not depend on the stored width
            first = a if first is None else first
            np.testing.assert_array_equal(a, first)
        eng.close()
