"""One scenario of tests/test_team_launch.py, in a process of its own: python launch_child.py SHIM SCENARIO.
The shim stands before the library's own launchers of the cooperative step."""
import ctypes
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path.insert(0, ROOT)
import __graft_entry__  # noqa: E402

__graft_entry__.load_package()
from sayram2d_gb300 import capi, cases  # noqa: E402

shim = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
LIB = capi.lib_path().encode()
FOREVER = 1 << 30


def shim_set(passed, refused):
    assert shim.shim_set(LIB, passed, refused) == 0


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


def refused_noalloc(passed):
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
        rc = capi.load().sayram_step_noalloc(ctypes.byref(s), None, 40, f.data_ptr(), out.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream, ctypes.byref(st))
        assert rc == capi.OK, capi.last_error()
        return out.cpu().numpy(), st.as_dict()

    capi.load()
    shim_set(FOREVER, 0)
    want = run()
    assert shim.shim_calls() == 2
    shim_set(passed, FOREVER)
    got = run()
    assert shim.shim_calls() == passed + 1
    assert np.array_equal(got[0], want[0]) and got[1] == want[1] and want[1]["steps"] == 40


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


SCENARIOS = {
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
