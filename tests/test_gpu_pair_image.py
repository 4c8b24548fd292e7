"""The float-pair images of the ephemeris files: only the own-time forces make
them, and not while their stream is being captured."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_other_calls_do_not_hold_a_second_copy_of_the_files(synth_files, tmp_path):
    """Body states, shared-time forces and a batch leave an ephemeris at little
    more than its files' size on the device (a float-pair image would double
    it)."""
    import torch
    from assist_gb300 import Ephem, batch, synth

    def use(pl, ast, system):
        e = Ephem(pl, ast)
        pop = synth.population(system, "mba", 64, seed=1, t0=8000.0)
        st = torch.tensor(pop.state, device="cuda")
        batch.bodies_device(e, torch.tensor([8000.0, 8001.0], dtype=torch.float64, device="cuda"))
        batch.forces_shared_time_device(e, 8000.0, st)
        t = torch.full((64,), 8000.0, dtype=torch.float64, device="cuda")
        batch.integrate_batch_device(e, t, t + 10.0, st)
        torch.cuda.synchronize()
        return e

    small = use(*synth_files)                       # loads the kernels and the scratch
    big = synth.write_ephemeris(str(tmp_path), seed=9, t_beg=7900.0, t_end=8100.0 + 120 * 365.25)
    size = os.path.getsize(big[0]) + os.path.getsize(big[1])
    assert size > 12 << 20
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    e = use(*big)
    used = free0 - torch.cuda.mem_get_info()[0]
    assert used < size + (8 << 20), (used, size)
    del small, e


def test_captured_own_time_forces(synth_files):
    """Own-time forces captured before and after the images exist: both replays
    give the accelerations (the bar of tests/test_gpu_forces.py), the second
    with the bits of a direct call."""
    import torch
    from assist_gb300 import Ephem, batch, synth
    from tests.oracle_py import Oracle
    pl, ast, system = synth_files
    n = 40
    pop = synth.population(system, "mix", n, seed=2, t0=8000.0)
    e = Ephem(pl, ast)
    t = 8000.0 + np.linspace(-20.0, 20.0, n)
    td, st = torch.tensor(t, device="cuda"), torch.tensor(pop.state, device="cuda")
    batch.bodies_device(e, td)                      # the ephemeris is on the device
    ref = np.array([Oracle(pl, ast).forces(t[i], pop.state[i:i + 1])[0] for i in range(n)])
    direct = None
    for _ in range(2):
        acc = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            batch.forces_device(e, td, st, acc=acc, stream=s)
        acc.zero_()
        g.replay()
        torch.cuda.synchronize()
        a = acc.cpu().numpy()
        assert (np.linalg.norm(a - ref, axis=1) < 1e-14 * np.linalg.norm(ref, axis=1)).all()
        if direct is not None:
            assert torch.equal(acc, direct)
        direct, _ = batch.forces_device(e, td, st)
        torch.cuda.synchronize()
