"""Particles that pass a planet deep inside its sphere of influence: the pilot
flags them whatever the batch's span, and the groups that hold one keep FP64
terms in every form of the batched call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T0 = 8000.0
BODY = {"Venus": (2, 2.45e-6, 0.006), "Earth": (3, 3.0e-6, 0.006), "Mars": (5, 3.2e-7, 0.005), "Jupiter": (6, 9.55e-4, 0.004)}


@pytest.fixture(scope="module")
def files(tmp_path_factory):
    from assist_gb300 import synth
    return synth.write_ephemeris(str(tmp_path_factory.mktemp("deep")), seed=8, t_beg=T0 - 100.0, t_end=T0 + 31 * 365.25)


def _path(O, t0, t1, state, tol=1e-11):
    """A path under the Sun and the planets as points of mass (their places from
    the oracle), by scipy's eighth-order Runge-Kutta."""
    from scipy.integrate import solve_ivp

    def f(t, y):
        a = np.zeros(3)
        for k in range(11):
            _, b = O.body(k, t)
            d = b[1:4] - y[:3]
            a += b[0] * d / (d @ d) ** 1.5
        return np.concatenate([y[3:], a])

    return solve_ivp(f, (t0, t1), state, method="DOP853", rtol=tol, atol=1e-13).y[:, -1]


def _flybys(files, share, when, seed):
    """States at T0 of particles that pass each planet at `share` of its radius
    of influence at the times `when`: from the pass backward.  Those whose path
    back is no moderate ellipse are drawn again."""
    from tests.oracle_py import Oracle
    pl, ast, system = files
    O = Oracle(pl, ast)
    rng = np.random.default_rng(seed)
    gms = 2.9591220828411951e-04
    out, names = [], []
    for name, (k, m, vinf) in BODY.items():
        for t in when:
            while True:
                p, v = system.body(k, np.array(t))
                s, sv = system.sun(np.array(t))
                d = share * np.linalg.norm(p - s) * m ** (1.0 / 3.0)
                u = rng.normal(size=3); u[2] *= 0.3; u /= np.linalg.norm(u)
                w = np.cross(u, rng.normal(size=3)); w /= np.linalg.norm(w)
                st = np.concatenate([p + d * u, v + np.sqrt(vinf ** 2 + 2.0 * m * gms / d) * w])
                pre = _path(O, t, t - 60.0, st)
                h = pre - np.concatenate(system.sun(np.array(t - 60.0)))
                a = 1.0 / (2.0 / np.linalg.norm(h[:3]) - h[3:] @ h[3:] / gms)
                e = np.linalg.norm(np.cross(h[3:], np.cross(h[:3], h[3:])) / gms - h[:3] / np.linalg.norm(h[:3]))
                if 0.0 < a < 20.0 and e < 0.7:
                    break
            out.append(_path(O, t - 60.0, T0, pre))
            names.append((name, t))
    return np.array(out), names


def _flags(eph, t0, te, state):
    import torch
    from assist_gb300 import batch
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    return batch.deep_pass_device(eph, dev(t0), dev(te), dev(state)).cpu().numpy()


@pytest.mark.parametrize("years", [1, 8, 30])
def test_deep_passes_are_flagged_whatever_the_span(files, years):
    """Passes at 0.02 of the radius of influence are flagged in batches of one
    to thirty years, early and late in them, in a short span inside a long
    batch too; a main belt is not, but for its few with such a pass."""
    from assist_gb300 import Ephem, synth
    pl, ast, system = files
    eph = Ephem(pl, ast)
    span = years * 365.25
    fly, names = _flybys(files, 0.02, T0 + span * np.array([0.3, 0.62, 0.95]), 10 + years)
    pop = synth.population(system, "mba", 2000, seed=years, t0=T0)
    state = np.concatenate([fly, pop.state])
    t0 = np.full(len(state), T0)
    flags = _flags(eph, t0, np.full(len(state), T0 + span), state)
    assert [x for x, f in zip(names, flags) if not f] == []
    assert flags[len(fly):].mean() < 0.01
    # the same passes in spans that end a day after them, inside the long batch
    te = np.full(len(state), T0 + span)
    te[:len(fly)] = [t + 1.0 for _, t in names]
    flags = _flags(eph, t0, te, state)
    assert [x for x, f in zip(names, flags) if not f] == []
    # and spans of a day around each pass, backward, between the samples of the long one
    from tests.oracle_py import Oracle
    O = Oracle(pl, ast)
    late = np.array([_path(O, T0, t + 0.5, f) for f, (_, t) in zip(fly, names)])
    t = np.array([t for _, t in names])
    flags = _flags(eph, np.concatenate([t + 0.5, t0[:5]]), np.concatenate([t - 0.5, te[-5:]]), np.concatenate([late, pop.state[:5]]))
    assert [x for x, f in zip(names, flags) if not f] == []


def _mixed(files, n, n_fly, days, seed):
    """n main-belt particles and n_fly unbound flybys of Jupiter at about 0.02
    AU (0.04 of its radius of influence)."""
    from assist_gb300 import synth
    pl, ast, system = files
    pop = synth.population(system, "mba", max(n, 1), seed=seed, t0=T0)
    jp, jv = system.body(6, np.array(T0))
    fly = [np.concatenate([jp + 0.3 * np.eye(3)[k % 3] + 0.02 * np.eye(3)[(k + 1) % 3], jv - 0.02 * np.eye(3)[k % 3]])
           for k in range(n_fly)]
    state = np.concatenate([pop.state[:n], np.array(fly).reshape(-1, 6)])
    return state, np.full(len(state), T0), np.full(len(state), T0 + days)


@pytest.mark.parametrize("how", ["log", "warm"])
def test_learned_and_logged_batches_keep_deep_groups_apart(files, how):
    """With the learned start or the logging of its pairs, too, groups with a
    deep pass are the FP64 kernel's, and every particle ends where the oracle
    puts it."""
    import torch
    from assist_gb300 import Ephem, batch, warm
    from assist_gb300._lib import clib
    from tests.oracle_py import Oracle
    pl, ast, _ = files
    state, t0, te = _mixed(files, 200, 5, 100.0, 4)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    st, status = dev(state), torch.full((len(state),), -1, dtype=torch.int32, device="cuda")
    warm.set_params(np.zeros(warm.n_params()))          # a correction of nothing
    x, t = torch.zeros((4096, 32), device="cuda"), torch.zeros((4096, 21), device="cuda")
    try:
        if how == "log":
            assert clib.assist_gb300_warm_set_log(x.data_ptr(), t.data_ptr(), 4096, 1) == 0
        batch.integrate_batch_device(Ephem(pl, ast), dev(t0), dev(te), st, status=status,
                                     opts=batch.options(warm_start=2 if how == "warm" else 0))
        torch.cuda.synchronize()
        assert batch.last_deep_groups() > 0
        assert how == "warm" or clib.assist_gb300_warm_log_count() > 0
    finally:
        clib.assist_gb300_warm_set_log(None, None, 0, 1)
    assert (status.cpu().numpy() == 0).all()
    ref = Oracle(pl, ast).integrate_batch(t0, te, state)
    d = np.abs(st.cpu().numpy()[:, :3] - ref[:, :3]).max(axis=1)
    assert d[:200].max() < 1e-12 and d.max() < 1e-9, (d[:200].max(), d.max())


@pytest.mark.parametrize("n,n_fly,nv,dense", [(300, 5, 0, False), (0, 5, 0, False), (300, 5, 6, False), (0, 40, 6, False),
                                              (300, 5, 0, True)])
def test_split_batches_and_their_plans(files, n, n_fly, nv, dense):
    """Batches of which some groups or all hold a deep pass, with and without
    variational particles: against the oracle; a plan's replays have the direct
    call's bits, and so has a direct call again; dense output ends in the end
    states."""
    import torch
    from assist_gb300 import Ephem, batch
    from tests.oracle_py import Oracle
    pl, ast, _ = files
    eph = Ephem(pl, ast)
    state, t0, te = _mixed(files, n, n_fly, 100.0, 5)
    m = len(state)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    flags = _flags(eph, t0, te, state)
    assert flags[n:].all() and not flags[:n].any()
    _, groups = batch.group_plan(t0, te, state)
    var = np.tile(np.eye(6)[None], (m, 1, 1)) if nv else None
    got = []
    for _ in range(2):
        st, vs = dev(state), dev(var) if nv else None
        status = torch.full((m,), -1, dtype=torch.int32, device="cuda")
        if dense:
            out = torch.empty((2 * m, 6), dtype=torch.float64, device="cuda")
            batch.integrate_batch_dense_device(eph, dev(t0), dev(te), st, torch.arange(0, 2 * m + 1, 2, dtype=torch.int32, device="cuda"),
                                               dev(np.tile([T0 + 50.0, T0 + 100.0], m)), out, status=status)
            assert torch.equal(out[1::2], st)
        else:
            batch.integrate_batch_device(eph, dev(t0), dev(te), st, var_state=vs, status=status)
        deep = batch.last_deep_groups()
        assert deep == sum(flags[g].any() for g in groups) and (deep == len(groups)) == (n == 0)
        assert (status.cpu().numpy() == 0).all()
        got.append((st, vs))
    assert torch.equal(got[0][0], got[1][0]) and (not nv or torch.equal(got[0][1], got[1][1]))
    ref = Oracle(pl, ast).integrate_batch(t0, te, state, var_state=var, return_all=True)
    d = np.abs(got[0][0].cpu().numpy()[:, :3] - ref[0][:, :3]).max(axis=1)
    assert d.max() < 1e-9 and (n == 0 or d[:n].max() < 1e-12), d.max()
    if nv:
        rel = np.abs(got[0][1].cpu().numpy() - ref[1]).max(axis=(1, 2)) / np.abs(ref[1]).max(axis=(1, 2))
        assert rel.max() < 1e-6, rel.max()
    if dense:
        return
    # a plan over the same particles
    a, b = dev(t0), dev(te)
    st, vs = dev(state), dev(var) if nv else None
    status = torch.full((m,), -1, dtype=torch.int32, device="cuda")
    plan = batch.Plan(eph, a, b, st, var_state=vs, status=status)
    assert batch.last_deep_groups() == deep
    for _ in range(3):
        st.copy_(dev(state))
        if nv:
            vs.copy_(dev(var))
        plan.launch()
        plan.stats()
        assert (status.cpu().numpy() == 0).all()
        assert torch.equal(st, got[0][0]) and (not nv or torch.equal(vs, got[0][1]))
    plan.close()


def test_step_limits_of_unequal_spans(files):
    """Satellites of the Earth, whose search ends at its step limit (1,000 and
    two a day), with spans from 30 to 440 days beside each other in a warp, and
    main-belt particles among them."""
    from assist_gb300 import Ephem, synth
    pl, ast, system = files
    ep, ev = system.body(3, np.array(T0))
    gm = 2.9591220828559115e-4 * 3.003e-6
    pop = synth.population(system, "mba", 24, seed=3, t0=T0)
    state, te = pop.state.copy(), np.full(24, T0 + 100.0)
    sat = np.arange(24) % 3 != 2
    for i in np.flatnonzero(sat):
        r = 0.0100 * (0.10 + 0.0007 * i)
        u, w = np.eye(3)[i % 3], np.eye(3)[(i + 1) % 3]
        state[i] = np.concatenate([ep + r * u, ev + (gm / r) ** 0.5 * w])
        te[i] = T0 + 30.0 + 17.8 * i
    flags = _flags(Ephem(pl, ast), np.full(24, T0), te, state)
    long = sat & (te - T0 > 200.0)
    assert flags[long].all() and not flags[~sat].any()


LEARNED = """
import sys
import numpy as np, torch
from assist_gb300 import Ephem, batch
from tests.test_gpu_deep import _mixed
from assist_gb300 import warm
pl, ast, out = sys.argv[1:4]
warm.set_params(np.zeros(warm.n_params()))          # a correction of nothing
d = np.load(out)
dev = lambda a: torch.tensor(a, device="cuda")
st = dev(d["state"])
status = torch.full((len(st),), -1, dtype=torch.int32, device="cuda")
batch.integrate_batch_device(Ephem(pl, ast), dev(d["t0"]), dev(d["te"]), st, status=status, opts=batch.options(warm_start=2))
torch.cuda.synchronize()
np.savez(out, state=st.cpu().numpy(), status=status.cpu().numpy(), deep=batch.last_deep_groups())
"""


def test_learned_batch_of_deep_groups_only(files, tmp_path):
    """The learned start with every group deep, in a process whose first batch
    this is: the workspace is this batch's alone."""
    import os
    import subprocess
    import sys
    from tests.oracle_py import Oracle
    pl, ast, _ = files
    state, t0, te = _mixed(files, 0, 40, 100.0, 5)
    f = str(tmp_path / "batch.npz")
    np.savez(f, state=state, t0=t0, te=te)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", LEARNED, pl, ast, f], check=True, cwd=root, timeout=300)
    got = np.load(f)
    assert (got["status"] == 0).all() and got["deep"] >= 2
    ref = Oracle(pl, ast).integrate_batch(t0, te, state)
    assert np.abs(got["state"][:, :3] - ref[:, :3]).max() < 1e-9
