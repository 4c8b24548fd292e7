"""Host threads with ephemerides of their own call the library at once."""
import struct
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _more_asteroids(path, out, extra):
    """The asteroid file with the first `extra` segments listed again under
    numbers of their own (without a mass)."""
    raw = bytearray(open(path, "rb").read())
    count = int(struct.unpack_from("<d", raw, 1024 + 16)[0])
    for k in range(extra):
        s = list(struct.unpack_from("<dd6i", raw, 1024 + 24 + 40 * k))
        s[2] = 2009000 + k
        struct.pack_into("<dd6i", raw, 1024 + 24 + 40 * (count + k), *s)
    struct.pack_into("<d", raw, 1024 + 16, float(count + extra))
    with open(out, "wb") as f:
        f.write(raw)
    return str(out)


def test_own_time_forces_from_threads_with_different_asteroid_counts(synth_files, tmp_path):
    """Two threads, one with 25 asteroids and one with 16, each call the
    own-time forces with variational particles on a stream of its own: no call
    fails, and every result has the bits of a call made alone (the block's
    dynamic shared memory grows with the asteroids, past 48 KB with 25; its
    limit is the kernel's, not the call's)."""
    import torch
    from assist_gb300 import Ephem, batch, synth
    pl, ast, system = synth_files
    n = 40
    pop = synth.population(system, "mix", n, seed=3, t0=8000.0)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    t, st = dev(8000.0 + np.linspace(-20.0, 20.0, n)), dev(pop.state)
    var = dev(np.tile(np.eye(6)[None], (n, 1, 1)))
    ephems = [Ephem(pl, _more_asteroids(ast, tmp_path / "more.bsp", 9)), Ephem(pl, ast)]
    alone = [batch.forces_device(e, t, st, var_state=var) for e in ephems]
    torch.cuda.synchronize()
    fail = [None, None]
    go = threading.Barrier(2)

    def work(k):
        s = torch.cuda.Stream()
        acc, vacc = torch.empty_like(alone[k][0]), torch.empty_like(alone[k][1])
        go.wait()
        try:
            for _ in range(8):
                for _ in range(1000):
                    batch.forces_device(ephems[k], t, st, var_state=var, acc=acc, var_acc=vacc, stream=s)
                s.synchronize()
                assert torch.equal(acc, alone[k][0]) and torch.equal(vacc, alone[k][1])
        except Exception as e:  # noqa: BLE001
            fail[k] = e

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for x in ts:
        x.start()
    for x in ts:
        x.join()
    assert fail == [None, None], fail
