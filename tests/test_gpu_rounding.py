"""The small terms' own rounding: what a term adds to an evaluation, and an
evaluation's whole error, against the oracle in double-double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EARTH_H, SUN_H, ALL = 0x10, 0x20, 0x7F
T = 8200.0
N = 1000
# Two evaluations that differ in one small term share every other operation
# but the roundings of the sums that it enters: at most two FP64 additions
# each, so four roundings of up to half an ulp, 2^-53 of the component,
# uniformly distributed.
DIFF_RMS = 2.0 * 2.0 ** -53 / 3.0 ** 0.5


@pytest.fixture(scope="module")
def world(tmp_path_factory):
    from assist_gb300 import Ephem, synth
    from tests.oracle_py import Oracle
    pl, ast, system = synth.write_ephemeris(str(tmp_path_factory.mktemp("round")), seed=6, t_beg=7950.0, t_end=8450.0)
    return Ephem(pl, ast), Oracle(pl, ast), system


def _around(system, body, lo, hi, seed):
    """N states at lo..hi AU from a body at T, moving with it on the whole."""
    rng = np.random.default_rng(seed)
    x, v = system.body(body, np.array(T))
    u = rng.normal(size=(N, 3))
    u *= rng.uniform(lo, hi, (N, 1)) / np.linalg.norm(u, axis=1, keepdims=True)
    return np.concatenate([x + u, v + 1e-3 * rng.normal(size=(N, 3))], axis=1)


def _gpu(eph, state, forces, kind):
    """acc (N, 3), or with kind "var" the derivatives by state too (N, 7, 3)."""
    import torch
    from assist_gb300 import batch
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    o = batch.options(forces=forces)
    if kind == "shared":
        return batch.forces_shared_time_device(eph, T, dev(state), opts=o).cpu().numpy()
    var = dev(np.tile(np.eye(6), (len(state), 1, 1))) if kind == "var" else None
    acc, vacc = batch.forces_device(eph, dev(np.full(len(state), T)), dev(state), var_state=var, opts=o)
    if var is None:
        return acc.cpu().numpy()
    return np.concatenate([acc.cpu().numpy()[:, None], vacc.cpu().numpy()], axis=1)


def _oracle(O, state, forces, kind, dd=True):
    if kind != "var":
        return O.forces(T, state, forces=forces, dd=dd)
    n = len(state)
    got = O.forces(T, state, var_state=np.tile(np.eye(6), (n, 1)), var_tp=np.repeat(np.arange(n), 6).astype(np.int32),
                   forces=forces, dd=dd)
    lay = lambda a: np.concatenate([a[:n, None], a[n:].reshape(n, 6, 3)], axis=1)  # noqa: E731
    return lay(got) if not dd else (lay(got[0]), lay(got[1]))


@pytest.mark.parametrize("kind,term,lo,hi", [
    ("shared", EARTH_H, 0.0205, 0.023), ("own", EARTH_H, 0.0205, 0.023), ("var", EARTH_H, 0.101, 0.12),
    ("shared", SUN_H, 0.101, 0.13), ("own", SUN_H, 0.101, 0.13), ("var", SUN_H, 0.101, 0.13),
    ("shared", SUN_H, 0.101, 0.499), ("var", SUN_H, 0.101, 0.499),
    ("shared", SUN_H, 0.501, 0.55), ("own", SUN_H, 0.501, 0.55), ("var", SUN_H, 0.501, 0.55)])
def test_harmonics_add_no_more_than_rounding(world, kind, term, lo, hi):
    """The harmonics beyond the distances within which they are FP64 (0.02 AU
    of the Earth, 0.1 with derivatives; 0.1 AU of the Sun) or float pairs (0.5
    AU of the Sun): what switching them on adds, against the double-double
    oracle."""
    eph, O, system = world
    state = _around(system, 3 if term == EARTH_H else 0, lo, hi, 1)
    got = _gpu(eph, state, ALL, kind) - _gpu(eph, state, ALL & ~term, kind)
    (ah, al), (bh, bl) = _oracle(O, state, ALL, kind), _oracle(O, state, ALL & ~term, kind)
    diff = got - ((ah - bh) + (al - bl))
    parts = [(diff, ah)]
    if kind == "var":
        # the acceleration, and the Jacobian by position
        parts = [(diff[:, 0], ah[:, 0]), (diff[:, 1:4].reshape(N, 9), ah[:, 1:4].reshape(N, 9))]
    for d, a in parts:
        e = np.linalg.norm(d, axis=1) / np.linalg.norm(a, axis=1)
        rms = np.sqrt((e ** 2).mean())
        print("%s: rms %.2e, bound %.2e" % (kind, rms, DIFF_RMS))
        assert rms < DIFF_RMS


@pytest.mark.parametrize("body,lo,hi", [(10, 0.45, 0.8), (5, 0.05, 0.2), (3, 0.08, 0.3), (11, 0.004, 0.05), (26, 0.001, 0.02)])
def test_derivatives_near_light_bodies(world, body, lo, hi):
    """The Jacobian by position about bodies whose pull is small beside the
    Sun's when their tidal field is not: its error is no more than twice the
    FP64 oracle's (whose square root and division round to half an ulp each
    where the kernels' reciprocal root has one)."""
    eph, O, system = world
    state = _around(system, body, lo, hi, 2)
    ref = _oracle(O, state, ALL, "var")

    def rms(x):
        e = ((x - ref[0]) - ref[1])[:, 1:4].reshape(N, 9)
        return np.sqrt(((np.linalg.norm(e, axis=1) / np.linalg.norm(ref[0][:, 1:4].reshape(N, 9), axis=1)) ** 2).mean())
    g, o = rms(_gpu(eph, state, ALL, "var")), rms(_oracle(O, state, ALL, "var", dd=False))
    print("body %d: rms %.2e, oracle %.2e" % (body, g, o))
    assert g < 2.0 * o


@pytest.mark.parametrize("kind", ["shared", "own", "var"])
def test_sums_round_once(world, kind):
    """The terms beside the Sun's enter the acceleration in one rounding: it
    differs from the Sun's alone by the double-double difference and two
    roundings, uniform over an ulp of each component (a tenth more for
    sampling and for the small terms' own rounding; a third would be 1.22)."""
    from assist_gb300 import synth
    eph, O, system = world
    state = synth.population(system, "mba", N, seed=8, t0=T, length=1.0).state
    one = 0x1
    a, b = _gpu(eph, state, ALL, kind), _gpu(eph, state, one, "own" if kind == "var" else kind)
    (ah, al), (bh, bl) = _oracle(O, state, ALL, "own"), _oracle(O, state, one, "own")
    e = ((a[:, 0] if kind == "var" else a) - b) - ((ah - bh) + (al - bl))
    expect = np.sqrt((2.0 * np.spacing(np.abs(ah)) ** 2 / 12.0).mean())
    rms = np.sqrt((e ** 2).mean())
    print("%s: rms %.3f of the expected" % (kind, rms / expect))
    assert rms < 1.1 * expect


# solar masses by ASSIST's body index: Mercury, Venus, Earth, Mars, Saturn, Uranus, Neptune (the bound has one close
# body: the Moon's neighbourhood is the Earth's too)
LIGHT = {1: 1.66e-7, 2: 2.45e-6, 3: 3.0e-6, 5: 3.2e-7, 7: 2.86e-4, 8: 4.37e-5, 9: 5.15e-5}


@pytest.mark.parametrize("kind", ["shared", "own"])
@pytest.mark.parametrize("body", sorted(LIGHT))
def test_close_bodies_in_fp64(world, kind, body):
    """Particles 0.02 to 0.7 of the way to a body's threshold, where its term
    has to be FP64's.  Bound of an error: four ulp of the body's and the
    particle's place, with the term's slope of 3, and 4e-16 of the whole; a
    float pair's 1.5e-15 of the place rms is 3.4 times the first."""
    eph, O, system = world
    m, (x, _) = LIGHT[body], system.body(body, np.array(T))
    R = np.linalg.norm(x)
    thr = max(m / 1e-3, (150 * m) ** (2 / 3)) ** 0.5 * R
    state = _around(system, body, 0.02 * thr, 0.7 * thr, 3)
    got = _gpu(eph, state, ALL, kind)
    h, l = _oracle(O, state, ALL, "own")
    d = np.linalg.norm(state[:, :3] - x, axis=1)
    pull = 2.9591220828559115e-4 * m / d ** 2
    a = np.linalg.norm(h, axis=1)
    bound = 3.0 * 4.0 * 2.0 ** -53 * R / d * pull + 4e-16 * a
    e = np.linalg.norm((got - h) - l, axis=1) / bound
    print("body %d %s: rms %.2f of the bound" % (body, kind, np.sqrt((e ** 2).mean())))
    assert np.sqrt((e ** 2).mean()) < 1.0
