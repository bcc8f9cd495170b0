"""What a handle holds after a call that failed: every particle its own last
valid position, type and caller index."""
import numpy as np
import pytest

from test_gpu_parity import _engine

pytestmark = pytest.mark.gpu


def _far(x, y, L):
    d = x - y
    d -= L * np.round(d / L)
    return np.abs(d).max()


@pytest.mark.parametrize("case", ["fluid", "patchy"])
def test_state_after_a_period_that_gave_up(case):
    """Chunks that give up inside a period (a neighbour's records never come)
    leave their particles where their last step put them, not the words of a
    buffer from before the last sort."""
    from pyrdsim_gb300 import abi, workloads
    from pyrdsim_gb300.engine import EngineError
    sd = (workloads.active_wall_fluid(n=8192, seed=3) if case == "fluid"
          else workloads.patchy_colloids(n_molecules=2048, seed=3))
    # (launches of an odd number of steps end in the other buffer)
    e = _engine([sd], sync_wait_ms=20, list_period=11)
    L = np.asarray(sd.model.L, dtype=float)
    e.step(10)
    x0, t0 = e.state()
    e.test_withhold(5)
    for steps in (13, 8):  # steps 11 to 21, a whole period; 24 to 30, part of one
        with pytest.raises(EngineError) as ei:
            e.step(steps)
        assert ei.value.code == abi.ERR_SYNC, str(ei.value)
        x, t = e.state()
        # at most the allowed displacement (half the skin) per period begun
        assert _far(x, x0, L) < 2 * 0.5 * e.info()["skin"], _far(x, x0, L)
        assert (t != t0).mean() < 0.01
        x0, t0 = x, t
    e.close()


@pytest.mark.parametrize("bad", ["nan", "outside", "type"])
def test_refused_state_changes_nothing(bad):
    """set_state with one bad entry is refused; state, neighbour pairs, g(r),
    observables and the steps after it are those of a handle that never saw it."""
    from pyrdsim_gb300.engine import EngineError
    from test_gpu_pairs import _fluid
    sd = _fluid(1501, 40.0, 2, (1, -1), 3.0, seed=5, types=2)
    e, ref = _engine([sd]), _engine([sd])
    for h in (e, ref):
        h.step(33)
    x, t = e.state()
    xb, tb = x[::-1].copy(), t[::-1].copy()  # other particles' places
    if bad == "nan":
        xb[700, 0] = np.nan
    elif bad == "outside":
        xb[700, 1] = 41.0
    else:
        tb[700] = 2
    with pytest.raises(EngineError):
        e.set_state(xb, tb)
    for steps in (0, 14):
        if steps:
            for h in (e, ref):
                h.step(steps)
        for a, b in zip(e.state(), ref.state()):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(e.pairs(), ref.pairs())
        np.testing.assert_array_equal(e.rdf_counts(9.0, 50), ref.rdf_counts(9.0, 50))
        np.testing.assert_array_equal(e.drift(), ref.drift())
        np.testing.assert_equal(e.observables(), ref.observables())
    e.close()
    ref.close()


@pytest.mark.parametrize("graphs", [True, False])
def test_pairs_use_their_cells_again_after_a_good_call(graphs):
    """After a device error pairs are looked for in every cell; a later call that
    rebuilds the cells and ends well makes that needless."""
    from pyrdsim_gb300.engine import EngineError
    from test_gpu_pairs import _distances, _fluid
    sd = _fluid(1024, 40.0, 2, (1, 1), 3.0, seed=6)
    e = _engine([sd], use_graphs=graphs, skin=0.04)
    xi = np.zeros((3, 1024, 2))
    xi[:, 5] = 10.0  # one particle moved by more than half the skin
    # (steps 4 to 13 fail too, up to the rebuild of step 10; 14 to 18 have none)
    for steps, every in ((0, 1), (10, 1), (5, 1), (20, 0)):
        if steps == 0:
            with pytest.raises(EngineError):
                e.step(3, xi=xi, u1=np.ones((3, 1024)), u2=np.ones((3, 1024)))
        elif steps == 10:
            with pytest.raises(EngineError):
                e.step(steps, noise=False)
        else:
            e.step(steps, noise=False)
        r = _distances(e.state()[0], 40.0, (1, 1))
        i, j = np.nonzero(np.triu(r <= 3.0, 1))
        np.testing.assert_array_equal(e.pairs(),
                                      np.stack([i, j], 1).astype(np.int32).reshape(-1, 2))
        assert e.test_lists()["every_cell"] == every, steps
    e.close()
