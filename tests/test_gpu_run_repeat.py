"""The drop-in's run kernels: repeats give the same bits, and a step past either
end of the ephemeris stops with the coverage error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def files(tmp_path_factory):
    from assist_gb300 import synth
    return synth.write_ephemeris(str(tmp_path_factory.mktemp("run")), seed=6, t_beg=7950.0, t_end=8250.0)


def _simulation(eph, state, var):
    from assist_gb300 import Extras, Simulation
    sim = Simulation.create()
    ex = Extras(sim, eph)
    for s in state:
        sim.add(*s)
    if var:
        for i in range(len(state)):
            for name in ("x", "y", "z", "vx", "vy", "vz"):
                setattr(sim.particle(sim.add_variation(i)), name, 1.0)
    sim.t = 8000.0
    return sim, ex


@pytest.mark.parametrize("n,t1,var", [(3, 8060.0, False), (100, 8060.0, False), (1025, 8030.0, False), (7, 8040.0, True),
                                      (40, 8030.0, True)])
def test_repeats_bit_for_bit(files, n, t1, var):
    """One block and several that meet at the grid barrier."""
    from assist_gb300 import Ephem, synth
    pl, ast, system = files
    eph = Ephem(pl, ast)
    pop = synth.population(system, "neo", n, seed=50 + n, t0=8000.0)
    out = []
    for _ in range(3):
        sim, ex = _simulation(eph, pop.state, var)
        assert sim.integrate(t1) == 0 and sim.t == t1
        out.append(np.array([[p.x, p.y, p.z, p.vx, p.vy, p.vz] for p in sim.particles]))
        ex.detach(sim); sim.free()
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("n,var", [(1, False), (33, False), (9, True)])
def test_past_the_ephemeris(files, n, var, sign):
    """Forward past its end and backward past its start: the coverage error,
    with the simulation short of the end and its states still numbers."""
    from assist_gb300 import Ephem, synth
    pl, ast, system = files
    pop = synth.population(system, "mba", n, seed=70 + n, t0=8000.0)
    sim, ex = _simulation(Ephem(pl, ast), pop.state, var)
    sim.integrate(8000.0 + sign * 10000.0)
    assert sim.status == 1
    assert 8000.0 < sim.t < 8300.0 if sign > 0 else 7900.0 < sim.t < 8000.0
    assert all(np.isfinite([p.x, p.y, p.z, p.vx, p.vy, p.vz]).all() for p in sim.particles)
    ex.detach(sim); sim.free()
