"""Particles far outside the planets, and states that are not numbers, with
variational particles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAR = (150.0, 250.0, 3e3, 1e5, 9e5, 2e6, 1e9, 1e13)      # either side of 200 AU and of 1e6 AU, where the terms' kinds change


@pytest.fixture(scope="module")
def files(tmp_path_factory):
    from assist_gb300 import synth
    return synth.write_ephemeris(str(tmp_path_factory.mktemp("far")), seed=6, t_beg=7950.0, t_end=8250.0)


def _far_states(rng):
    out = []
    for far in FAR:
        u = rng.normal(size=3); u /= np.linalg.norm(u)
        out.append(np.concatenate([far * u, 1e-2 * u[::-1]]))
    return np.array(out)


def test_own_time_forces_with_variational_far_out(files):
    """Accelerations and their derivatives by state against the oracle (the
    bar of tests/test_gpu_forces.py, 1e-14), and a state that is not a number
    gives none, without touching its neighbours."""
    import torch
    from assist_gb300 import Ephem, batch
    from tests.oracle_py import Oracle
    pl, ast, _ = files
    rng = np.random.default_rng(3)
    state = _far_states(rng)
    n = len(state)
    state = np.concatenate([state, state[:2]])
    state[n, 0] = np.nan
    state[n + 1, 4] = np.nan
    t = 8100.0 + rng.uniform(-100, 100, n + 2)
    var = rng.normal(size=(n + 2, 6, 6))
    var[:, :, :3] *= np.linalg.norm(state[:, None, :3], axis=2)[:, :, None]     # position's and velocity's shares both count
    var[n:] = rng.normal(size=(2, 6, 6))
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    status = torch.full((n + 2,), -1, dtype=torch.int32, device="cuda")
    acc, vacc = batch.forces_device(Ephem(pl, ast), dev(t), dev(state), var_state=dev(var), status=status)
    acc, vacc = acc.cpu().numpy(), vacc.cpu().numpy()
    assert (status.cpu().numpy() == 0).all()
    O = Oracle(pl, ast)
    worst = 0.0
    for i in range(n):
        ref = O.forces(t[i], state[i:i + 1], var_state=var[i], var_tp=np.zeros(6, np.int32))
        e = np.linalg.norm(acc[i] - ref[0]) / np.linalg.norm(ref[0])
        d = np.linalg.norm(vacc[i] - ref[1:], axis=1).max() / np.linalg.norm(ref[1:], axis=1).max()
        print("far %g: acceleration %.2e derivatives %.2e" % (FAR[i], e, d))
        worst = max(worst, e, d)
    assert worst < 1e-14
    assert np.isnan(acc[n:]).all() and np.isnan(vacc[n]).all()


@pytest.mark.parametrize("n", [12, 40, 300])
def test_integrations_with_variational_far_out(files, n):
    """Far particles and one that is not a number among ordinary ones: in a
    batch each ends where the oracle puts it and only that one is marked; in a
    simulation (without the latter) likewise."""
    from assist_gb300 import Ephem, Extras, Simulation, batch, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    eph, O = Ephem(pl, ast), Oracle(pl, ast)
    pop = synth.population(system, "mba", n, seed=n, t0=8000.0)
    state = np.concatenate([pop.state, _far_states(np.random.default_rng(n))])
    m = len(state)
    bad = state.copy()
    bad[5, 1] = np.nan
    var = np.tile(np.eye(6)[None], (m, 1, 1))
    t0, te = np.full(m, 8000.0), np.full(m, 8060.0)
    out, vout, status, _ = batch.integrate_batch(eph, t0, te, bad, var_state=var)
    good = np.arange(m) != 5
    ref, vref, _, _ = O.integrate_batch(t0, te, state, var_state=var, return_all=True)
    scale = np.maximum(1.0, np.abs(ref[:, :3]).max(axis=1))
    assert status[5] == 2 and (status[good] == 0).all()
    assert (np.abs(out[good, :3] - ref[good, :3]).max(axis=1) / scale[good]).max() < 1e-12
    assert (np.abs(vout - vref).max(axis=(1, 2)) / np.abs(vref).max(axis=(1, 2)))[good].max() < 1e-9
    sim = Simulation.create(); ex = Extras(sim, eph)
    for s in state:
        sim.add(*s)
    for i in range(m):
        for k, name in enumerate(("x", "y", "z", "vx", "vy", "vz")):
            setattr(sim.particle(sim.add_variation(i)), name, 1.0)
    sim.t = 8000.0
    sim.integrate(8060.0)
    g = np.array([[p.x, p.y, p.z, p.vx, p.vy, p.vz] for p in sim.particles])
    tp = np.repeat(np.arange(m, dtype=np.int32), 6)
    r, rv, info = O.integrate(8000.0, 8060.0, state, var_state=np.tile(np.eye(6), (m, 1)), var_tp=tp)
    assert sim.status == 0 and info["status"] == 0
    assert (np.abs(g[:m, :3] - r[:, :3]).max(axis=1) / scale).max() < 1e-12
    assert (np.abs(g[m:] - rv).max(axis=1) / np.abs(rv).max(axis=1)).max() < 1e-9
    ex.detach(sim); sim.free()
