"""Scheduling slots of the one-state-per-thread kernels (fp64_tps, mixed_tps): 256
per handle, drawn by launch and put back by its last warp.  Many launches in a
row, ragged sizes and two streams at once reproduce a one-shot result bit for
bit; the layouts' shared-memory limits are the same for mechanisms of any size,
from any thread."""
import threading

import numpy as np
import pytest

from create_rate_subs_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _states(rs, n, seed):
    N = rs.n_species
    T, P, Y = synth.make_states(N, n, seed=seed)
    return tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1]))


@pytest.mark.parametrize("mode", ["fp64_tps", "mixed_tps"])
def test_slots_reused_and_two_streams(mode, synth_mech):
    from create_rate_subs_gb300.rates import RateSubs
    rs = RateSubs(synth_mech("gri53"))
    n = 20011
    T, P, Y = _states(rs, n, 41)
    want = rs.wdot(T, P, Y, mode=mode).clone()
    out = torch.empty_like(want)
    sizes = [1, 31, 32, 33, 317, 1000, n]
    for it in range(300):  # every slot is drawn again
        m = sizes[it % len(sizes)]
        out.fill_(float("nan"))
        rs.wdot(T[:m], P[:m], Y[:, :m], mode=mode, out=out[:, :m])
        if it % 37 == 0 or m == n:
            torch.cuda.synchronize()
            assert torch.equal(out[:, :m], want[:, :m]), (it, m)
    outs = [torch.full_like(want, float("nan")) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for it in range(20):
        for s, o in zip(streams, outs):
            with torch.cuda.stream(s):
                rs.wdot(T, P, Y, mode=mode, out=o)
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, want)
    assert rs.status()[0] == 0


@pytest.mark.parametrize("mode", ["fp64_strict", "fp64_tps", "fp64_warp", "fp64_tile", "mixed_tps",
                                  "mixed_warp", "mixed_tile"])
def test_two_mechanisms_from_two_threads(mode, synth_mech):
    """Each thread's launches have the shared memory that they ask for, whatever
    the other's mechanism needs."""
    from create_rate_subs_gb300.rates import RateSubs
    names = ["small", "large561" if "tile" in mode or "warp" in mode else "gri53"]
    errors, jobs = [], []
    for k, name in enumerate(names):
        rs = RateSubs(synth_mech(name))
        d = _states(rs, 97, k)
        jobs.append((rs, d, rs.wdot(*d, mode=mode), torch.cuda.Stream()))
    torch.cuda.synchronize()

    def work(job):
        rs, d, want, stream = job
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(stream):
                outs = [rs.wdot(*d, mode=mode) for _ in range(200)]
            stream.synchronize()
            assert all(torch.equal(o, want) for o in outs[::20])
        except Exception as e:  # reported by the test
            errors.append(e)
    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
