"""One scenario of tests/test_team_launch.py, in a process of its own: python launch_child.py SHIM SCENARIO.
The shim stands before the library's own launchers of the cooperative step."""
import ctypes
import os
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path.insert(0, ROOT)
import __graft_entry__  # noqa: E402

__graft_entry__.load_package()
from sayram2d_gb300 import capi, cases  # noqa: E402

shim = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
LIB = capi.lib_path().encode()
FOREVER = 1 << 30


def shim_set(passed, odd, give_up=0):
    assert shim.shim_set(LIB, passed, odd, give_up) == 0


def one(nx, ny, seed=3):
    return [cases.synthetic_problem(nx, ny, 1e-2, seed=seed, tau=0.7)]


def result(b):
    return [b.f(k) for k in range(len(b))], [b.stats(k) for k in range(len(b))]


def same(a, b):
    assert all(np.array_equal(x, y) for x, y in zip(a[0], b[0]))
    assert a[1] == b[1], (a[1], b[1])
    assert all(s["status"] == capi.OK for s in a[1])


def stepped(probs, prec, steps, coop, timing=False):
    b = capi.Batch(probs, precision=prec)
    b.set_coop(coop)
    b.enable_timing(timing)
    for n in steps:
        b.step(n)
    out = result(b)
    calls = shim.shim_calls()
    b.close()
    return out, calls


def refused(passed, probs, steps, timing=False):
    """The first launch but `passed` and all after it are refused: the steps are taken all the same, with
    the bits of the separate kernels, and the refused batch is not launched that way again."""
    for prec in (0, 1, 2):
        shim_set(0, 0)
        want, calls = stepped(probs, prec, steps, False)
        assert calls == 0
        shim_set(passed, FOREVER)
        got, calls = stepped(probs, prec, steps, True, timing)
        assert calls == passed + 1, calls
        same(got, want)


def noalloc_run(nsteps):
    """A call of the allocation-free step on one problem, as a function of nothing."""
    import torch

    p = one(64, 60)[0]
    keep = []

    def dev(a):
        keep.append(torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda"))
        return ctypes.cast(keep[-1].data_ptr(), capi._dp)

    s = capi.sayram_problem()
    s.nx, s.ny, s.dt = p.nx, p.ny, p.dt
    for name in ("x_edges", "y_edges", "G", "Dxx", "Dxy", "Dyy", "inv_tau"):
        setattr(s, name, dev(getattr(p, name)))
    s.f0 = capi._dp()
    for side in range(4):
        s.bc[side] = p.bc[side]
        s.dirichlet[side] = capi._dp() if p.dirichlet[side] is None else dev(p.dirichlet[side])
    f, st = torch.tensor(p.f0, device="cuda"), capi.sayram_stats()

    def run():
        out = torch.empty_like(f)
        rc = capi.load().sayram_step_noalloc(ctypes.byref(s), None, nsteps, f.data_ptr(), out.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream, ctypes.byref(st))
        return rc, out.cpu().numpy(), st.as_dict()

    run.keep = keep
    return run


def refused_noalloc(passed):
    run = noalloc_run(40)
    capi.load()
    shim_set(FOREVER, 0)
    want = run()
    assert shim.shim_calls() == 2
    shim_set(passed, FOREVER)
    got = run()
    assert shim.shim_calls() == passed + 1
    assert got[0] == want[0] == capi.OK and np.array_equal(got[1], want[1])
    assert got[2] == want[2] and want[2]["steps"] == 40


def refused_server():
    reqs = [(one(a, e, seed=a)[0], n) for a, e, n in ((40, 33, 7), (96, 80, 12), (17, 23, 5))]

    def serve():
        srv = capi.Server(2e9, max_slots=8, max_side=128, precision=2, lanes=2, split_side=64)
        ids = [srv.submit(*r) for r in reqs]
        for _ in range(100):
            srv.tick()
            if srv.info()["completed"] == len(reqs):
                break
        out = [srv.poll(i)[:2] for i in ids]
        srv.close()
        return [o[0] for o in out], [o[1] for o in out]

    capi.load()
    shim_set(FOREVER, 0)
    want = serve()
    shim_set(0, FOREVER)
    got = serve()
    assert shim.shim_calls() == 2  # once per lane
    same(got, want)


def fresh(probs, fs, prec, steps):
    """The batch's f after steps from the given states, by a batch that has seen nothing else."""
    b = capi.Batch(probs, precision=prec)
    for k, f in enumerate(fs):
        b.set_f(k, f)
    b.step(steps)
    out = result(b)[0]
    b.close()
    return out


def gave_up():
    """A wait that runs out loses the state of the batch: nothing is stepped on from it or read from it until
    every instance has a new one, launches queued behind it leave a lost instance alone, and then all is as in a
    new batch."""
    L = capi.load()
    probs = one(90, 70) + one(1, 1)  # a team of many blocks, and one of a single block, which waits for nobody
    fs = [np.array(p.f0) * 0.5 for p in probs]
    packed = np.concatenate([f.ravel() for f in fs])
    out = np.empty_like(packed)
    for prec in (0, 1, 2):
        shim_set(FOREVER, 0)
        want = fresh(probs, fs, prec, 3)
        b = capi.Batch(probs, precision=prec)
        b.step(2)
        its = b.stats(0)["total_iterations"]
        shim_set(0, 1, 1)
        assert L.sayram_batch_step(b.h, 70) == capi.ERR_TIMEOUT
        assert shim.shim_calls() == 3
        st = [b.stats(k) for k in range(2)]
        assert [s["status"] for s in st] == [capi.ERR_TIMEOUT] * 2
        assert st[0]["steps"] == 2 and st[0]["total_iterations"] == its, st
        m5, r = np.empty((5, 6300)), np.empty(6300)

        def refusals():
            return (L.sayram_batch_step(b.h, 1), L.sayram_batch_step_host(b.h, 1, None, out.ctypes.data),
                    L.sayram_batch_autotune(b.h, 1, None, None))

        assert refusals() == (capi.ERR_STATE,) * 3
        assert L.sayram_batch_get_f(b.h, 0, capi._ptr(out)) == capi.ERR_STATE
        assert L.sayram_batch_export_system(b.h, 0, capi._ptr(m5), capi._ptr(r)) == capi.ERR_STATE
        b.set_f(0, fs[0])
        assert np.allclose(b.f(0), fs[0], rtol=1e-14, atol=0) and refusals() == (capi.ERR_STATE,) * 3
        b.set_f(1, fs[1])
        assert b.stats(1)["status"] == capi.OK
        b.step(3)
        got = result(b)
        assert all(np.array_equal(x, y) for x, y in zip(got[0], want))
        assert all(s["status"] == capi.OK for s in got[1])
        # again, with the new states in the packed form
        shim_set(0, 1, 1)
        assert L.sayram_batch_step_host(b.h, 1, packed.ctypes.data, out.ctypes.data) == capi.ERR_TIMEOUT
        b.step_host(3, packed.ctypes.data, out.ctypes.data)
        assert np.array_equal(out, np.concatenate([f.ravel() for f in want]))
        b.close()


def gave_up_split():
    L = capi.load()
    probs = one(700, 620)
    for prec in (1, 2):
        shim_set(FOREVER, 0)
        want = fresh(probs, [probs[0].f0], prec, 2)
        b = capi.Batch(probs, precision=prec)
        b.step(2)
        shim_set(1, 1, 1)
        assert L.sayram_batch_step(b.h, 4) == capi.ERR_TIMEOUT
        assert b.stats(0)["steps"] == 3  # the first of the four
        b.set_f(0, probs[0].f0)
        b.step(2)
        assert np.array_equal(b.f(0), want[0])
        b.close()


def gave_up_autotune():
    """Tuning restores the state, whatever its steps came to."""
    L = capi.load()
    a, b = capi.Batch(one(90, 70), precision=2), capi.Batch(one(90, 70), precision=2)
    shim_set(FOREVER, 0)
    for x in (a, b):
        x.step(3)
    for passed in (0, 1):
        shim_set(passed, 1, 1)
        assert L.sayram_batch_autotune(a.h, 2, None, None) == capi.ERR_TIMEOUT
    for x in (a, b):
        x.step(3)
    assert np.array_equal(a.f(0), b.f(0))
    a.close()
    b.close()


def gave_up_noalloc():
    run = noalloc_run(40)
    capi.load()
    shim_set(FOREVER, 0)
    want = run()
    shim_set(0, 1, 1)
    assert run()[0] == capi.ERR_TIMEOUT
    got = run()
    assert got[0] == capi.OK and np.array_equal(got[1], want[1]) and got[2] == want[2]


def gave_up_server():
    L = capi.load()
    reqs = [(one(a, e, seed=a)[0], n) for a, e, n in ((40, 33, 7), (96, 80, 3), (17, 23, 5))]
    shim_set(FOREVER, 0)
    srv = capi.Server(2e9, max_slots=8, max_side=128, precision=2)

    def serve():
        ids = [srv.submit(*r) for r in reqs]
        for _ in range(7):
            srv.tick()
        return [srv.poll(i)[:2] for i in ids]

    want = serve()
    ids = [srv.submit(*r) for r in reqs]
    shim_set(2, 1, 1)
    srv.tick()
    srv.tick()
    n = ctypes.c_int()
    assert L.sayram_server_tick(srv.h, ctypes.byref(n)) == capi.ERR_TIMEOUT and n.value == 3
    info = srv.info()
    assert info["resident"] == 0 and info["arena_cells_used"] == 0 and info["completed"] == 6
    for i in ids:
        f, st = srv.poll(i)[:2]
        assert st["status"] == capi.ERR_TIMEOUT and np.isnan(f).all()
    got = serve()
    srv.close()
    for x, y in zip(got, want):
        assert np.array_equal(x[0], y[0]) and x[1] == y[1]


def side_by_side():
    """While another thread's call is in flight a launch takes at most half the SMs, and all of them again
    after it, with the same bits; a call in flight goes on with fewer when another begins."""
    import torch

    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    for prec in (0, 1, 2):
        for probs in (one(200, 180), cases.batch_problems(nsm + 8, 7, 1e-2, 8, 40)):
            shim_set(FOREVER, 0)
            other, alone, b = capi.Batch(one(33, 32), precision=prec), capi.Batch(probs, precision=prec), None
            alone.step(2)
            alone.step(2)
            whole = shim.shim_grid()
            assert nsm // 2 < whole <= nsm
            b = capi.Batch(probs, precision=prec)
            shim.shim_hold(400)
            t = threading.Thread(target=other.step, args=(1,))
            t.start()
            while not shim.shim_held():
                time.sleep(0.001)
            b.step(2)
            assert 0 < shim.shim_grid() <= nsm // 2, shim.shim_grid()
            t.join()
            time.sleep(0.05)
            b.step(2)
            assert shim.shim_grid() == whole
            same(result(b), result(alone))
            for x in (other, alone, b):
                x.close()


def beside_separate_kernels():
    """A call that runs as separate kernels is in flight like any other, in each of its forms."""
    import torch

    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    shim_set(FOREVER, 0)
    b = capi.Batch(one(200, 180), precision=2)
    b.step(1)
    whole = shim.shim_grid()
    a = capi.Batch(cases.batch_problems(24, 7, 1e-2, 64, 200), precision=2)
    a.set_launch_shape(4096, 32)  # segments too coarse for teams
    packed = np.concatenate([np.array(p.f0).ravel() for p in a.problems])
    out = np.empty_like(packed)
    for call in (lambda: a.step(2000), lambda: a.step_host(2000, packed.ctypes.data, out.ctypes.data),
                 lambda: a.autotune(200)):
        t = threading.Thread(target=call)
        t.start()
        time.sleep(0.1)
        b.step(1)
        grid = shim.shim_grid()
        assert t.is_alive()
        assert 0 < grid <= nsm // 2 < whole, (grid, whole)
        t.join()
        a.set_launch_shape(4096, 32)
    a.close()
    b.close()


SCENARIOS = {
    "side by side": side_by_side,
    "beside separate kernels": beside_separate_kernels,
    "gave up": gave_up,
    "gave up split": gave_up_split,
    "gave up autotune": gave_up_autotune,
    "gave up noalloc": gave_up_noalloc,
    "gave up server": gave_up_server,
    "first": lambda: refused(0, one(90, 70), (2, 1)),
    "second": lambda: refused(1, one(90, 70), (40, 1)),
    "bins": lambda: refused(0, cases.batch_problems(160, 7, 1e-2, 8, 40), (2,)),
    "split": lambda: refused(1, one(700, 620), (3, 1)),
    "timing": lambda: refused(0, one(90, 70), (2, 1), timing=True),
    "noalloc first": lambda: refused_noalloc(0),
    "noalloc second": lambda: refused_noalloc(1),
    "server": refused_server,
}

if __name__ == "__main__":
    SCENARIOS[sys.argv[2]]()
    print("scenario ok")
