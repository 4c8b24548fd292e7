"""The evaluation with pair terms (assist_gb300/csrc/fast_forces.cuh) at its
edges, against the oracle: group remainders, several groups a block, particles
on either side of every body's threshold and beyond FP32's range, no
asteroids; and a batch whose groups are split between the two kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-14          # the acceleration bar of tests/test_gpu_forces.py
MASS = {0: 1.66e-7, 1: 2.45e-6, 2: 3.0e-6, 3: 3.7e-8, 4: 3.2e-7, 5: 2.86e-4, 6: 4.4e-5, 7: 5.2e-5, 8: 7.4e-9}


@pytest.fixture(scope="module")
def files(tmp_path_factory):
    from assist_gb300 import synth
    return synth.write_ephemeris(str(tmp_path_factory.mktemp("fast")), seed=5, t_beg=7950.0, t_end=8450.0)


@pytest.mark.parametrize("n,asteroids", [(1, True), (31, True), (33, True), (33, False), (15000, True)])
def test_shared_time_forces_at_thresholds(files, n, asteroids):
    import torch
    from assist_gb300 import Ephem, batch, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    eph = Ephem(pl, ast if asteroids else "/nonexistent")
    t = 8100.25
    pop = synth.population(system, "mix", n, seed=n, t0=t, nongrav_frac=0.3)
    rng = np.random.default_rng(n)
    extra = []
    for k in range(9):                      # on either side of each pair body's threshold
        body = system.body(k + 1 if k < 5 else k + 2, np.array(t))
        thr = max(MASS[k] / 1e-3, (150 * MASS[k]) ** (2 / 3)) ** 0.5
        for f in (0.7, 0.95, 1.05):
            u = rng.normal(size=3); u /= np.linalg.norm(u)
            extra.append(np.concatenate([body[0] + f * thr * np.linalg.norm(body[0]) * u, body[1]]))
    for far in (2e6, 1e9, 1e13):            # beyond the range of the FP32 products
        u = rng.normal(size=3); u /= np.linalg.norm(u)
        extra.append(np.concatenate([far * u, 1e-2 * u[::-1]]))
    state = np.concatenate([pop.state, np.array(extra)])
    params = np.concatenate([pop.params, np.zeros((len(extra), 3))])
    st, prm = torch.tensor(state, device="cuda"), torch.tensor(params, device="cuda")
    status = torch.full((len(state),), -1, dtype=torch.int32, device="cuda")
    acc = batch.forces_shared_time_device(eph, t, st, params=prm, status=status).cpu().numpy()
    assert (status.cpu().numpy() == 0).all()
    idx = np.arange(len(state)) if n < 1000 else np.concatenate([np.arange(0, n, 97), np.arange(n - 40, len(state))])
    ref = Oracle(pl, ast if asteroids else "/nonexistent").forces(t, state[idx], params=params[idx])
    e = np.linalg.norm(acc[idx] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert e.max() < TOL, (e.max(), idx[e.argmax()])


def test_batch_split_between_kernels(files):
    """Particles that pass Jupiter well inside its sphere of influence share a
    batch with ordinary ones: every particle ends where the oracle puts it."""
    import torch
    from assist_gb300 import Ephem, batch, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    eph = Ephem(pl, ast)
    pop = synth.population(system, "mba", 100, seed=9, t0=8000.0, length=100.0)
    jp, jv = system.body(6, np.array(8000.0))
    fly = []
    for k in range(5):                      # unbound flybys of Jupiter at about 0.02 AU
        u, w = np.eye(3)[k % 3], np.eye(3)[(k + 1) % 3]
        fly.append(np.concatenate([jp + 0.3 * u + 0.02 * w, jv - 0.02 * u]))
    state = np.concatenate([pop.state, np.array(fly)])
    n = len(state)
    t0, te = np.full(n, 8000.0), np.full(n, 8100.0)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    st, status = dev(state), torch.full((n,), -1, dtype=torch.int32, device="cuda")
    batch.integrate_batch_device(eph, dev(t0), dev(te), st, status=status)
    assert (status.cpu().numpy() == 0).all()
    ref = Oracle(pl, ast).integrate_batch(t0, te, state)
    d = np.abs(st.cpu().numpy()[:, :3] - ref[:, :3]).max(axis=1)
    assert d[:100].max() < 1e-12 and d.max() < 1e-9, (d[:100].max(), d.max())


@pytest.mark.parametrize("n,t1", [(1, 8100.0), (32, 7960.0), (33, 8100.0), (300, 8060.0)])
def test_dropin_run_kernel(files, n, t1):
    """Shared-step simulations of one block and several, forward and backward,
    against the oracle; one integration in two calls ends where one call does
    to rounding, and a step past the ephemeris stops with the coverage error."""
    from assist_gb300 import Ephem, Extras, Simulation, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    eph = Ephem(pl, ast)
    pop = synth.population(system, "mba", n, seed=n, t0=8000.0)

    def run(stops):
        sim = Simulation.create(); ex = Extras(sim, eph)
        for s in pop.state:
            sim.add(*s)
        sim.t = 8000.0
        for t in stops:
            sim.integrate(t)
        g = np.array([[p.x, p.y, p.z] for p in sim.particles])
        out = sim.status, sim.t, sim.steps_done, g
        ex.detach(sim); sim.free()
        return out

    st, t, steps, g = run([t1])
    ref, _, info = Oracle(pl, ast).integrate(8000.0, t1, pop.state)
    assert st == 0 and t == t1 and abs(steps - info["accepted"]) <= 1
    assert np.abs(g - ref[:, :3]).max() < 1e-13
    st, t, _, g2 = run([0.5 * (8000.0 + t1), t1])
    assert st == 0 and t == t1 and np.abs(g2 - g).max() < 1e-13
    st, t, _, _ = run([t1, 20000.0])
    assert st == 1 and t < 8500.0 or t1 < 8000.0


@pytest.mark.parametrize("n", [1, 33, 1024, 1025, 1100])
def test_bodies_bit_identical(files, n):
    """Both body kernels (few times, many times; remainders of a tile) give the
    oracle's bits, which are the reference's."""
    import torch
    from assist_gb300 import Ephem, batch
    from tests.oracle_py import Oracle
    pl, ast, _ = files
    t = np.random.default_rng(n).uniform(7960.0, 8440.0, n)
    status = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    B = batch.bodies_device(Ephem(pl, ast), torch.tensor(t, device="cuda"), status=status).cpu().numpy()
    assert (status.cpu().numpy() == 0).all()
    O = Oracle(pl, ast)
    for k in range(0, n, max(1, n // 40)):
        for i in range(27):
            _, ref = O.body(i, t[k])
            m = 10 if i < 11 else 4
            assert np.array_equal(B[k, i, :m], ref[:m]), (k, i, B[k, i, :m] - ref[:m])
            assert i < 11 or np.isnan(B[k, i, 4:]).all()


@pytest.mark.parametrize("n,var", [(1, False), (31, True), (33, False), (70, True)])
def test_own_time_forces_at_thresholds(files, n, var):
    """Each particle at its own time: tile remainders, particles on either side
    of the pair bodies' thresholds and of the harmonics', and (accelerations)
    beyond FP32's range; a time outside the ephemeris marks its particle only."""
    import torch
    from assist_gb300 import Ephem, batch, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    t0 = 8200.0
    rng = np.random.default_rng(n)
    pop = synth.population(system, "mix", n, seed=n, t0=t0, nongrav_frac=0.3)
    extra, te = [], []
    for k in range(9):
        for f in (0.7, 1.3, 1.5):
            t = t0 + rng.uniform(-100, 100)
            body = system.body(k + 1 if k < 5 else k + 2, np.array(t))
            thr = max(MASS[k] / 1e-3, (150 * MASS[k]) ** (2 / 3)) ** 0.5
            u = rng.normal(size=3); u /= np.linalg.norm(u)
            extra.append(np.concatenate([body[0] + f * thr * np.linalg.norm(body[0]) * u, body[1]])); te.append(t)
    for b, d in ((3, 0.03), (3, 0.09), (3, 0.11), (0, 0.08), (0, 0.12)):
        body = system.body(b, np.array(t0))
        u = rng.normal(size=3); u /= np.linalg.norm(u)
        extra.append(np.concatenate([body[0] + d * u, body[1] + 1e-2 * u[::-1]])); te.append(t0)
    if not var:
        for far in (300.0, 2e6, 1e13):
            u = rng.normal(size=3); u /= np.linalg.norm(u)
            extra.append(np.concatenate([far * u, 1e-2 * u[::-1]])); te.append(t0)
    state = np.concatenate([pop.state, np.array(extra)])
    tt = np.concatenate([t0 + rng.uniform(-100, 100, n), te])
    params = np.concatenate([pop.params, np.zeros((len(extra), 3))])
    vs = rng.normal(size=(len(state), 6, 6)) if var else None
    dev = lambda a: None if a is None else torch.tensor(a, device="cuda")  # noqa: E731
    eph, O = Ephem(pl, ast), Oracle(pl, ast)
    status = torch.full((len(state),), -1, dtype=torch.int32, device="cuda")
    acc, vacc = batch.forces_device(eph, dev(tt), dev(state), params=dev(params), var_state=dev(vs), status=status)
    assert (status.cpu().numpy() == 0).all()
    acc = acc.cpu().numpy()
    for i in range(len(state)):
        kw = dict(var_state=vs[i], var_tp=np.zeros(6, np.int32)) if var else {}
        ref = O.forces(tt[i], state[i:i + 1], params=params[i:i + 1], **kw)
        assert np.linalg.norm(acc[i] - ref[0]) < TOL * np.linalg.norm(ref[0]), (i, np.linalg.norm(acc[i] - ref[0]) / np.linalg.norm(ref[0]))
        if var:
            scale = np.linalg.norm(ref[1:], axis=1).max()
            d = np.linalg.norm(vacc[i].cpu().numpy() - ref[1:], axis=1).max()
            assert d <= TOL * scale, (i, d / scale)
    tt[0] = 20000.0
    _, _ = batch.forces_device(eph, dev(tt), dev(state), params=dev(params), var_state=dev(vs), status=status)
    s = status.cpu().numpy()
    assert s[0] == 5 and (s[1:] == 0).all()


def test_batch_repeats_bit_for_bit(files):
    """The builds of the batched kernel, and one build run again, give the same
    bits (their warps share the state across barriers)."""
    import torch
    from assist_gb300 import Ephem, batch, synth
    pl, ast, system = files
    eph = Ephem(pl, ast)
    pop = synth.population(system, "neo", 6000, seed=4, t0=8000.0, length=200.0, nongrav_frac=0.2)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    t0, te, prm = dev(pop.t0), dev(pop.t_end), dev(pop.params)
    out = []
    for kw in (dict(blocks_per_sm=2), dict(blocks_per_sm=2), dict(blocks_per_sm=3), dict(ephem_staging=1)):
        st = dev(pop.state)
        batch.integrate_batch_device(eph, t0, te, st, params=prm, opts=batch.options(**kw))
        out.append(st.cpu().numpy())
    assert all(np.array_equal(out[0], o) for o in out[1:])


@pytest.mark.parametrize("n,t1", [(1, 8060.0), (9, 8060.0), (70, 8030.0), (2440, 8003.0)])
def test_dropin_run_kernel_with_variational(files, n, t1):
    """Six variational particles a particle, their slots dealt in a shuffled
    order: one block, two with a remainder of one, nine, and more particles
    than blocks of eight fit on the device (sixteen a block)."""
    from assist_gb300 import Ephem, Extras, Simulation, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    pop = synth.population(system, "neo", n, seed=31, t0=8000.0)
    tp = np.repeat(np.arange(n, dtype=np.int32), 6)
    var0 = np.tile(np.eye(6), (n, 1))
    mix = np.random.default_rng(n).permutation(6 * n)
    tp, var0 = np.ascontiguousarray(tp[mix]), np.ascontiguousarray(var0[mix])
    sim = Simulation.create(); ex = Extras(sim, Ephem(pl, ast))
    for s in pop.state:
        sim.add(*s)
    for k in range(6 * n):
        p = sim.particle(sim.add_variation(int(tp[k])))
        p.x, p.y, p.z, p.vx, p.vy, p.vz = var0[k]
    sim.t = 8000.0
    sim.integrate(t1)
    assert sim.status == 0 and sim.t == t1
    g = np.array([[p.x, p.y, p.z, p.vx, p.vy, p.vz] for p in sim.particles])
    r, rv, info = Oracle(pl, ast).integrate(8000.0, t1, pop.state, var_state=var0, var_tp=tp)
    assert info["status"] == 0
    assert np.abs(g[:n, :3] - r[:, :3]).max() < 1e-9
    rel = np.abs(g[n:] - rv).max(axis=1) / np.abs(rv).max(axis=1)
    assert rel.max() < 1e-7
    assert abs(sim.steps_done - info["accepted"]) <= 1
    ex.detach(sim); sim.free()


@pytest.mark.parametrize("n,length,sign", [(1, 60.0, 1.0), (16, 60.0, 1.0), (33, 60.0, -1.0), (20500, 2.0, 1.0),
                                           (27000, 1.0, 1.0)])
def test_batch_with_variational(files, n, length, sign):
    """Batches with six variational particles each, a third with
    non-gravitational parameters, of unequal lengths, forward and backward:
    one group, remainders of groups of sixteen, many of those, and more than
    they are formed for (samples of those against the oracle)."""
    from assist_gb300 import Ephem, batch, synth
    from tests.oracle_py import Oracle
    pl, ast, system = files
    pop = synth.population(system, "mix", n, seed=40 + n, t0=8000.0, nongrav_frac=0.34)
    rng = np.random.default_rng(n)
    t0 = np.full(n, 8000.0)
    te = t0 + sign * length * rng.uniform(0.1, 1.0, n)
    var = np.tile(np.eye(6)[None], (n, 1, 1)) + 1e-3 * rng.standard_normal((n, 6, 6))
    out, vout, status, _ = batch.integrate_batch(Ephem(pl, ast), t0, te, pop.state, params=pop.params, var_state=var)
    i = np.arange(n) if n < 1000 else np.arange(0, n, 83)
    ref, vref, rstat, _ = Oracle(pl, ast).integrate_batch(t0[i], te[i], pop.state[i], params=pop.params[i], var_state=var[i],
                                                          return_all=True)
    assert (status == 0).all() and (rstat == 0).all()
    assert np.abs(out[i, :3] - ref[:, :3]).max() < 1e-9
    rel = np.abs(vout[i] - vref).max(axis=(1, 2)) / np.abs(vref).max(axis=(1, 2))
    assert rel.max() < 1e-7
