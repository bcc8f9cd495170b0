"""The period kernel (one launch per graph-replayed rebuild period, CTAs
synchronised by the progress words of neighbouring chunks) against the
per-step drift and reaction kernels it replaces: identical states bit for bit
(same per-particle arithmetic), and a wait that runs out ends the call with
RDSIM_ERR_SYNC instead of hanging the GPU."""
import numpy as np
import pytest

from test_gpu_parity import _case, _engine

pytestmark = pytest.mark.gpu


def _workload(case):
    from pyrdsim_gb300 import workloads
    if case == "active_wall_fluid_65536":
        # fast reactions: several listed draws per chunk and step
        return [workloads.active_wall_fluid(n=65536, seed=5, k_on=2.0, k_off=5.0)]
    if case == "active_wall_fluid_rx":
        return [workloads.active_wall_fluid(n=4096, seed=7, k_on=20.0, k_off=50.0)]
    if case == "patchy_colloids":
        return [workloads.patchy_colloids(n_molecules=2048, seed=3)]
    if case == "lj_fluid":
        return [workloads.lj_fluid(n=1024, seed=1, start="lattice")]
    if case == "ensemble":
        return workloads.ensemble(n_systems=8, n_min=256, n_max=4096, seed=11)
    return [_case(case)[1]]


CASES = ["active_wall_fluid_65536", "active_wall_fluid_rx", "patchy_colloids", "lj_fluid",
         "ensemble", "two_species_wall_rx", "patchy", "mixed_laws", "lj3d"]


@pytest.mark.parametrize("case", CASES)
def test_period_kernel_is_bit_identical(case):
    """Positions, types and drift equal those of the per-step kernels after
    calls that start, split and end rebuild periods."""
    sds = _workload(case)
    one = _engine(sds)
    per_step = _engine(sds, period_kernel=False)
    assert one.info()["period_kernel"] == 1, one.info()
    assert per_step.info()["period_kernel"] == 0
    prev = one.state()[1]
    changed = 0
    for n in (5, 33, 64, 1, 97):
        one.step(n)
        per_step.step(n)
        xa, ta = one.state()
        xb, tb = per_step.state()
        np.testing.assert_array_equal(ta, tb)
        np.testing.assert_array_equal(xa, xb)
        changed += int((ta != prev).sum())
        prev = ta
    np.testing.assert_array_equal(one.drift(), per_step.drift())
    if case in ("active_wall_fluid_65536", "active_wall_fluid_rx", "two_species_wall_rx"):
        assert changed >= 5, "too few reactions to exercise the listed draws"


def test_period_kernel_replaces_the_step_launches():
    """A replayed period is six launches (five rebuild kernels and the period
    kernel) instead of five plus two per step."""
    from pyrdsim_gb300 import workloads
    sd = workloads.active_wall_fluid(n=8192, seed=3)
    e = _engine([sd])
    e.step(9)  # reach the start of a period
    e.profile()
    e.step(41)  # steps 10..50
    prof = e.profile()
    # periods 10, 20, 30 and 40 replayed (one period kernel each), the last
    # step 50 by its own drift kernel
    assert prof["force"]["launches"] == 4 + 1, prof


def test_period_wait_runs_out_without_hanging():
    """A chunk that never publishes its progress makes its neighbours' waits
    end after the limit: the call returns RDSIM_ERR_SYNC, the handle stays
    usable, and once restored it steps like a fresh handle."""
    from pyrdsim_gb300 import abi, workloads
    from pyrdsim_gb300.engine import EngineError
    sd = workloads.active_wall_fluid(n=8192, seed=3)
    e = _engine([sd], sync_wait_ms=20)
    x0, t0 = e.state()
    e.step(9)
    e.test_withhold(5)
    with pytest.raises(EngineError) as ei:
        e.step(25)
    assert ei.value.code == abi.ERR_SYNC, str(ei.value)
    assert "waited longer" in str(ei.value)
    e.test_withhold(-1)
    e.set_state(x0, t0)
    e.step_index = 0
    ref = _engine([sd])
    ref.set_state(x0, t0)  # the same float64 round trip of the state
    for n in (9, 25):
        e.step(n)
        ref.step(n)
    xa, ta = e.state()
    xb, tb = ref.state()
    np.testing.assert_array_equal(ta, tb)
    np.testing.assert_array_equal(xa, xb)


@pytest.mark.parametrize("case", ["lj_fluid", "patchy_colloids", "active_wall_fluid_rx"])
def test_list_period_keeps_results(case):
    """A list period longer than the deck's rebuild frequency (larger skin,
    fewer rebuilds) gives the same dynamics: identical types and positions
    within 1e-6 after 60 steps with injected noise (float32 pair sums in
    another order), and the period kernel equals the per-step kernels bit
    for bit at that period too."""
    sds = _workload(case)
    n = sum(s.n_particles for s in sds)
    D = sds[0].model.N_dim
    rng = np.random.default_rng(4)
    xi = rng.standard_normal((60, n, D))
    u1 = np.ones((60, n))  # no reaction fires: decisions cannot sit on a threshold
    ref = _engine(sds)
    longp = _engine(sds, list_period=30)
    assert longp.info()["skin"] > ref.info()["skin"]
    ref.step(60, xi=xi, u1=u1, u2=u1)
    longp.step(60, xi=xi, u1=u1, u2=u1)
    xa, ta = ref.state()
    xb, tb = longp.state()
    np.testing.assert_array_equal(ta, tb)
    L = np.asarray(sds[0].model.L[:D], dtype=float)
    d = xb - xa
    d -= L * np.round(d / L)
    assert np.abs(d).max() <= 1e-6 * max(1.0, np.abs(xa).max()), np.abs(d).max()
    a, b = ref.drift(), longp.drift()
    assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(a)
    one = _engine(sds, list_period=30)
    per_step = _engine(sds, list_period=30, period_kernel=False)
    for k in (7, 64, 30):
        one.step(k)
        per_step.step(k)
    np.testing.assert_array_equal(one.state()[0], per_step.state()[0])
    np.testing.assert_array_equal(one.state()[1], per_step.state()[1])


def test_period_kernel_fallbacks_are_exact():
    """A long list period (large skin: rows longer than the 32 staged entries,
    chunks whose neighbour runs overflow the staging table) mixes staged and
    gathered particles within CTAs; the period kernel still equals the
    per-step kernels bit for bit."""
    from pyrdsim_gb300 import workloads
    sd = workloads.active_wall_fluid(n=8192, seed=9, k_on=20.0, k_off=50.0)
    one = _engine([sd], list_period=80)
    per_step = _engine([sd], list_period=80, period_kernel=False)
    assert one.info()["period_kernel"] == 1 and one.info()["list_width"] > 32
    for n in (79, 250, 3, 170):  # four 80-step periods run as period kernels
        one.step(n)
        per_step.step(n)
        xa, ta = one.state()
        xb, tb = per_step.state()
        np.testing.assert_array_equal(ta, tb)
        np.testing.assert_array_equal(xa, xb)
    np.testing.assert_array_equal(one.drift(), per_step.drift())


@pytest.mark.parametrize("n", [2, 15, 17, 1000, 14593, 29191, 30011])
def test_period_lanes_and_frames(n):
    """The period kernel's lanes per chain follow the number of particles (4,
    2 and 1 here); launches also end before trajectory frames and the call's
    last step.  Positions, types, frames and drifts equal the per-step
    kernels' bit for bit at every size, with ragged last chunks and calls that
    start and end inside list periods."""
    from pyrdsim_gb300 import workloads
    # (a handful of particles at the fluid's density would fill a box smaller
    # than the interaction range)
    sd = workloads.active_wall_fluid(n=n, rho=0.4 if n >= 1000 else 0.02, seed=n, k_on=20.0,
                                     k_off=50.0)
    one = _engine([sd])
    per_step = _engine([sd], period_kernel=False)
    assert one.info()["period_kernel"] == 1
    for e in (one, per_step):
        e.set_trajectory(7, 6)
    for k in (3, 44, 1, 2, 25):
        one.step(k)
        per_step.step(k)
        for a, b in zip(one.state() + one.trajectory(), per_step.state() + per_step.trajectory()):
            np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(one.drift(), per_step.drift())
    np.testing.assert_array_equal(one.reaction_rates(), per_step.reaction_rates())


@pytest.mark.parametrize("n", [1, 63, 65, 4099, 250001])
def test_lj_walk_equals_the_general_walk(n):
    """A large system whose pair laws are all Lennard-Jones n = 6 takes the drift
    kernel's Lennard-Jones walk; adding a law between types that no particle
    has sends it through the general one.  Drifts and states are the same bit
    for bit, with rows within and beyond the stored list width."""
    from pyrdsim_gb300 import model, workloads
    sd = workloads.inhibited_mixture(n=n, seed=n, rho=0.45 if n >= 1000 else 0.02)
    m = sd.model
    p = dict(m.parameters)
    p["tau_by_taud"] = np.ones(4)
    p["interactions"] = list(m.interactions) + [
        {"type": "yukawa", "pair": [3, 3], "u0": 1.0, "r0": 0.5, "rc": 1.1}]
    general = model.SystemData(model.Model.from_dict(p), sd.x, sd.types, sd.molecule_ids,
                               sd.first_index)
    for width in (0, 8):
        es = [_engine([s], period_kernel=False, list_width=width) for s in (sd, general)]
        for k in (1, 30):
            for e in es:
                e.step(k)
            for a, b in zip(es[0].state(), es[1].state()):
                np.testing.assert_array_equal(a, b)
            np.testing.assert_array_equal(es[0].drift(), es[1].drift())


@pytest.mark.parametrize("n,D,width", [(1, 2, 0), (16, 2, 0), (17, 2, 8), (65, 2, 0), (1100, 2, 0),
                                       (2049, 3, 0), (2060, 3, 8), (70, 1, 0)])
def test_list_builder_of_small_and_3d_systems(n, D, width):
    """Rows built by 16 lanes per particle, at remainders of a chunk and with rows
    beyond the stored width: the drift from them against float64 (the suite's
    bounds), and the period kernel's states from the codes written with them
    against the per-step kernels' from the rows."""
    from test_gpu_force64 import _system
    from test_gpu_parity import _oracle, drift_errors
    sd = _system(n, D, "lj")
    one = _engine([sd], list_width=width)
    norm, per = drift_errors(one.drift(), _oracle(sd).drift())
    assert norm < 1e-5 and per < 1e-4, (norm, per)
    steps = _engine([sd], list_width=width, period_kernel=False)
    for k in (23, 12):
        one.step(k)
        steps.step(k)
        np.testing.assert_array_equal(one.state()[0], steps.state()[0])


@pytest.mark.parametrize("n,D", [(2048, 2), (2049, 2), (1331, 3), (1100, 1)])
def test_small_sort_equals_the_general_one(n, D):
    """Up to 2,048 particles one CTA sorts the cells; a batch with a second
    system takes the four kernels for both.  A system's rows, states and drift
    are the same bit for bit, with list builders of either form."""
    from pyrdsim_gb300 import model
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1.0 / D)))
    L = 1.5 * side
    g = np.stack(np.meshgrid(*[np.arange(side)] * D, indexing="ij"), -1).reshape(-1, D)
    x = (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.1, 0.1, (n, D))) * 1.5
    m = model.Model.from_dict({
        "n_dim": D, "l": np.full(D, L), "periodic": np.array([1.0] * (D - 1) + [-1.0]),
        "dt": 1e-4, "n_steps": 10, "n_out": 1000, "tau_by_taud": np.ones(2), "seed": 3,
        "interactions": [{"type": "lj", "pair": [a, b], "u0": 1.0, "r0": 1.1, "rc": 2.5, "n": 6}
                         for a, b in ((0, 0), (0, 1), (1, 1))],
        "reactions": [{"type": "linear", "reactant": 0, "product": 1, "rate": 20.0},
                      {"type": "locally_catalyzed", "reactant": 1, "catalyst": 0, "product": 0,
                       "rate": 20.0, "r0": 1.6}]})
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    sd = model.SystemData(m, x, rng.integers(0, 2, n).astype(np.int32), mol,
                          np.arange(n, dtype=np.int32))
    alone, batch = _engine([sd]), _engine([sd, sd])
    for k in (25, 8, 13):
        alone.step(k)
        batch.step(k)
        (xa, ta), (xb, tb) = alone.state(), batch.state()
        np.testing.assert_array_equal(xa, xb[:n])
        np.testing.assert_array_equal(ta, tb[:n])
    np.testing.assert_array_equal(alone.drift(), batch.drift()[:n])
