"""Scratch of the state tiles (net rates that do not fit on chip): launches on
any streams, from any threads and in any graphs of one handle run side by side,
each with blocks of its own."""
import ctypes
import threading

import numpy as np
import pytest

from create_rate_subs_gb300 import _lib, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# sizes with scratch: three CTAs per SM; clusters and a CTA per SM of a mechanism
# whose rates do not fit on chip
CASES = [("gri53", 153 * 32 + 1, "fp64"), ("gri53", 20000, "mixed"), ("large561", 700, "fp64"),
         ("large561", 33, "mixed"), ("large561", 5000, "fp64")]


def _states(mech, n, seed):
    N = mech.n_species
    T, P, Y = synth.make_states(N, n, seed=seed)
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]


@pytest.mark.parametrize("name,n,mode", CASES)
def test_many_streams_and_threads(name, n, mode, synth_mech):
    from create_rate_subs_gb300.rates import RateSubs
    mech = synth_mech(name)
    rs = RateSubs(mech)
    sets = [_states(mech, n, s) for s in range(4)]
    want = [rs.wdot(*d, mode=mode) for d in sets]
    streams = [torch.cuda.Stream() for _ in range(12)]
    outs = [torch.empty_like(want[0]) for _ in streams]
    torch.cuda.synchronize()

    def work(part):
        for _ in range(6):
            for k in part:
                with torch.cuda.stream(streams[k]):
                    rs.wdot(*sets[k % 4], mode=mode, out=outs[k])
    threads = [threading.Thread(target=work, args=(range(k, 12, 3),)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for k, o in enumerate(outs):
        assert torch.equal(o, want[k % 4])


@pytest.mark.parametrize("name,n,mode", CASES)
def test_graph_instantiated_twice_and_cloned(name, n, mode, synth_mech):
    """A captured first call, its graph instantiated twice and cloned, all three
    launched at the same time: no node of the graph is tied to one executable."""
    from create_rate_subs_gb300.rates import RateSubs
    mech = synth_mech(name)
    d = _states(mech, n, 3)
    want = RateSubs(mech).wdot(*d, mode=mode)
    rs = RateSubs(mech)
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        rs.wdot(*d, mode=mode, out=out)
    cu = ctypes.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc
    graph, clone = ctypes.c_void_p(g.raw_cuda_graph()), ctypes.c_void_p()
    ok(cu.cuGraphClone(ctypes.byref(clone), graph))
    execs = []
    for src in (graph, graph, clone):
        e = ctypes.c_void_p()
        ok(cu.cuGraphInstantiateWithFlags(ctypes.byref(e), src, ctypes.c_ulonglong(0)))
        execs.append(e)
    streams = [torch.cuda.Stream() for _ in execs]
    for _ in range(5):
        for e, s in zip(execs, streams):
            ok(cu.cuGraphLaunch(e, ctypes.c_void_p(s.cuda_stream)))
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    out.zero_()
    ok(cu.cuGraphLaunch(execs[2], ctypes.c_void_p(streams[2].cuda_stream)))
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    for e in execs:
        ok(cu.cuGraphExecDestroy(e))
    ok(cu.cuGraphDestroy(clone))


def test_first_call_while_another_thread_captures(synth_mech):
    """The scratch is made on the first call: also while a capture elsewhere
    forbids allocations by default."""
    from create_rate_subs_gb300.rates import RateSubs
    mech = synth_mech("gri53")
    n = 153 * 32 + 1
    d = _states(mech, n, 5)
    want = RateSubs(mech).wdot(*d)
    rs, lib = RateSubs(mech), _lib.load()
    out, out2 = torch.zeros_like(want), torch.zeros_like(want)
    side, result = torch.cuda.Stream(), []
    torch.cuda.synchronize()

    def work():
        torch.cuda.set_device(0)
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        result.append(lib.crs_wdot(rs.h, n, p(d[0]), p(d[1]), p(d[2]), n, p(out),
                                   _lib.MODES["fp64"], ctypes.c_void_p(side.cuda_stream)))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        t = threading.Thread(target=work)
        t.start()
        t.join()
        out2.copy_(want)
    assert result == [0], _lib.last_error()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out2, want)
