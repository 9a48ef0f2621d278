"""The cooperative step (whole steps in one launch, a team of blocks per instance) against the separate
kernels of the same step: the two share their formulas, reduction segments and orders of summation, so
states and statistics must agree bit for bit at every split of the work. Also the other paths that
hand work to it, at the sizes where they change form."""
import ctypes
import dataclasses

import numpy as np
import pytest

from sayram2d_gb300 import cases

pytestmark = pytest.mark.gpu


def _run(capi, probs, prec, precond, coop, calls):
    b = capi.Batch(probs, precision=prec, precond=precond)
    b.set_coop(coop)
    l0 = b.launches()
    for n in calls:
        b.step(n)
    used = b.launches() - l0
    out = [b.f(k) for k in range(len(probs))]
    stats = [b.stats(k) for k in range(len(probs))]
    b.close()
    return out, stats, used


def _same(a, b):
    for k, (x, y) in enumerate(zip(a[0], b[0])):
        assert np.array_equal(x, y), (k, x.shape, float(np.abs(x - y).max()))
    for k, (x, y) in enumerate(zip(a[1], b[1])):
        assert x == y, (k, x, y)


# cells per reduction segment: 128 up to 65,536 cells (rows padded to 4), 256 up to 131,072, 512 up to
# 262,144, then 1024; a cell per lane in the smallest shares; a separate assembly launch from 2048 cells
# per block; the vectors leave the chip above 4096 (FP64) or 8192 cells per block
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("nx,ny,precond", [
    (1, 1, 1), (33, 32, 1), (33, 32, 0), (1, 513, 1), (5, 700, 0), (700, 5, 1), (2500, 40, 1),
    (260, 252, 1), (260, 253, 0), (389, 517, 1), (640, 410, 1), (700, 620, 0), (900, 880, 1)])
def test_one_instance(capi, nx, ny, precond, prec):
    p = cases.synthetic_problem(nx, ny, 1e-2, seed=nx + ny, tau=0.7)
    team = _run(capi, [p], prec, precond, True, (2, 1))
    _same(team, _run(capi, [p], prec, precond, False, (2, 1)))
    assert all(s["status"] == 0 for s in team[1])
    # a few launches of it, not one per pass
    assert team[2] <= 4 * 3, team[2]


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("nx,ny,dt", [(900, 880, 1e-5), (389, 517, 1e-4), (700, 620, 1e-3)])
def test_solves_of_one_iteration_with_chunks_in_turn(capi, nx, ny, dt, prec):
    """Short time steps end a solve after one iteration, whose residual pass reads the shadow residual in
    the neighbouring chunks' rows while it writes the next one: with one block per SM a chunk's
    neighbours are written long before or after it reads them."""
    p = cases.synthetic_problem(nx, ny, dt, seed=nx, tau=0.7)
    got = []
    for coop in (True, False, False):
        b = capi.Batch([p], precision=prec, inner_tol=1e-2, max_refine=40)
        b.set_launch_shape(1024, 1)
        b.set_coop(coop)
        b.step(3)
        got.append(([b.f(0)], [b.stats(0)]))
        b.close()
    _same(got[0], got[1])
    _same(got[1], got[2])
    s = got[0][1][0]
    assert s["status"] == 0
    if dt == 1e-5:  # some solves took one iteration
        assert s["total_iterations"] < 2 * (s["total_refinements"] - s["steps"]), s


@pytest.mark.parametrize("prec", [1, 2])
def test_one_instance_between_two_and_eight_thousand_cells_a_block(capi, prec):
    """1.3 million cells: by their number they would take chunks of 4096, but the step still fits the
    cooperative form, with vectors in global memory."""
    p = cases.synthetic_problem(1180, 1100, 1e-2, seed=5, tau=0.7)
    b = capi.Batch([p], precision=prec)
    assert b.launch_shape()[0] == 2048
    b.close()
    team = _run(capi, [p], prec, 1, True, (2,))
    _same(team, _run(capi, [p], prec, 1, False, (2,)))
    assert team[2] <= 4 * 2, team[2]


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n,lo,hi", [(24, 20, 220), (40, 100, 200), (152, 8, 60), (153, 8, 60), (400, 1, 48)])
def test_many_instances(capi, n, lo, hi, prec):
    """Teams of several blocks, one block each, and (more instances than SMs) several per block."""
    probs = cases.batch_problems(n, 7, 1e-2, lo, hi)
    team = _run(capi, probs, prec, 1, True, (2,))
    _same(team, _run(capi, probs, prec, 1, False, (2,)))
    assert team[2] <= 4 * 2, team[2]


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_steps_of_one_call_equal_single_calls(capi, prec):
    """More steps than one launch takes."""
    p = [cases.synthetic_problem(48, 40, 1e-2, seed=3, tau=0.7)]
    a = _run(capi, p, prec, 1, True, (70,))
    b = _run(capi, p, prec, 1, True, (1,) * 70)
    _same(a, b)


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("nx", [479, 480, 960])
def test_dirichlet_values_of_any_number(capi, nx, prec):
    """A side's values travel 480 to a launch: 480, 481 and 961 of them, as if set at creation."""
    p = cases.synthetic_problem(nx, 6, 1e-2, seed=nx, tau=0.7)
    side = next(s for s in (2, 3) if p.dirichlet[s] is not None)
    v = np.linspace(0.25, 1.75, nx + 1) * np.asarray(p.dirichlet[side]).max()
    q = dataclasses.replace(p, dirichlet=[v if s == side else d for s, d in enumerate(p.dirichlet)])
    a, b = capi.Solver(p, precision=prec), capi.Solver(q, precision=prec)
    a.set_dirichlet(side, v)
    a.step(2)
    b.step(2)
    fa, fb = a.f(), b.f()
    a.close()
    b.close()
    assert np.array_equal(fa, fb)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 70), (33, 29), (129, 65)])
def test_state_in_and_out(capi, nx, ny, prec):
    """set_f then f: FP64 as it is, double-word rounded to hi + lo."""
    p = cases.synthetic_problem(nx, ny, 1e-2, seed=9, tau=0.7)
    f = np.random.default_rng(nx).uniform(0.0, 1.0, (nx, ny)) * 10.0 ** np.random.default_rng(ny).uniform(-30, 30, (nx, ny))
    s = capi.Solver(p, precision=prec)
    s.set_f(f)
    got = s.f()
    s.close()
    hi = f.astype(np.float32)
    want = f if prec != 2 else hi.astype(np.float64) + (f - hi).astype(np.float32).astype(np.float64)
    assert np.array_equal(got, want)


def test_noalloc_grid_too_wide_for_the_chip(capi, oracle):
    """Rows so long that a block's vectors with both halo rows do not fit: pass by pass, to the same
    tolerance as the other forms (1e-10 in relative L2)."""
    torch = pytest.importorskip("torch")
    nx, ny = 4000, 16
    p = cases.synthetic_problem(nx, ny, 1e-2, seed=31, tau=0.7)
    keep = {}

    def dev(a):
        keep[len(keep)] = torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")
        return ctypes.cast(keep[len(keep) - 1].data_ptr(), capi._dp)

    s = capi.sayram_problem()
    s.nx, s.ny, s.dt = nx, ny, p.dt
    for name in ("x_edges", "y_edges", "G", "Dxx", "Dxy", "Dyy", "inv_tau"):
        setattr(s, name, dev(getattr(p, name)))
    s.f0 = capi._dp()
    for side in range(4):
        s.bc[side] = p.bc[side]
        s.dirichlet[side] = capi._dp() if p.dirichlet[side] is None else dev(p.dirichlet[side])
    f = torch.tensor(p.f0, device="cuda")
    out = torch.empty_like(f)
    st = capi.sayram_stats()
    rc = capi.load().sayram_step_noalloc(ctypes.byref(s), None, 2, f.data_ptr(), out.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream, ctypes.byref(st))
    assert rc == capi.OK, capi.last_error()
    got, ref = out.cpu().numpy(), oracle.step(p, None, 2, solver="splu")
    assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
    assert st.steps == 2 and got.min() >= 0.0


@pytest.mark.parametrize("lanes", [1, 2])
def test_server_regions_taken_again(capi, lanes):
    """Requests served from regions that held others give the bits of a fresh server's."""
    def requests(seed, sizes):
        return [(cases.synthetic_problem(a, e, 1e-2, seed=seed + k, tau=0.5), 3 + k) for k, (a, e) in enumerate(sizes)]

    def serve(srv, reqs):
        ids = [srv.submit(*r) for r in reqs]
        for _ in range(100):
            srv.tick()
            if srv.info()["resident"] == 0 and srv.info()["waiting"] == 0:
                break
        return [srv.poll(i)[0] for i in ids]

    first = requests(1, [(120, 90), (33, 20), (64, 64), (20, 130)])
    second = requests(50, [(70, 111), (128, 128), (9, 14), (40, 41)])
    kw = dict(max_slots=8, max_side=160, precision=2, lanes=lanes, split_side=64)
    a, b = capi.Server(5e8, **kw), capi.Server(5e8, **kw)
    serve(a, first)
    got, want = serve(a, second), serve(b, second)
    a.close()
    b.close()
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("coop", [True, False])
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("state", ["residual", "inf", "nan"])
def test_a_residual_out_of_range_is_not_converged(capi, state, prec, coop):
    """The sum of squares of a residual far above the right-hand side overflows FP32 (time step 1e25,
    boundary values 0: R is about 1e-28, R - M f about 1e-3), and a state that is not finite has no
    residual: no step may report either as solved. FP64 holds the first one's squares and solves it."""
    p = cases.synthetic_problem(24, 20, 1e25 if state == "residual" else 1e-2, seed=1, tau=1e30)
    p = dataclasses.replace(p, dirichlet=[None if d is None else 0.0 * np.asarray(d) for d in p.dirichlet])
    s = capi.Solver(p, precision=prec)
    s.set_coop(coop)
    f = np.array(p.f0)
    if state != "residual":
        f[5, 7] = float(state)
    s.set_f(f)
    rc = capi.load().sayram_update(s.h)
    st = s.stats(0)
    s.close()
    want = capi.OK if state == "residual" and prec == 0 else capi.ERR_NOT_CONVERGED
    assert rc == want and st["status"] == want, (rc, st)
    assert (st["rel_residual"] < 1e-10) == (want == capi.OK)


def test_handles_stepped_side_by_side(capi):
    """Handles of all kinds stepped from eight threads, in calls of one step and of many, with a server
    beside them: each gives the bits it gives alone, whatever share of the chip its launches had."""
    import threading

    kinds = [([cases.synthetic_problem(33, 32, 1e-2, seed=1, tau=0.7)], 0, (1,) * 40),
             ([cases.synthetic_problem(90, 90, 1e-2, seed=2, tau=0.7)], 0, (100,)),
             ([cases.synthetic_problem(80, 80, 1e-2, seed=3, tau=0.7)], 2, (1,) * 60),
             ([cases.synthetic_problem(389, 517, 1e-2, seed=4, tau=0.7)], 2, (40, 1, 1)),
             ([cases.synthetic_problem(700, 620, 1e-2, seed=5, tau=0.7)], 1, (3,) * 10),
             ([cases.synthetic_problem(256, 256, 1e-2, seed=6, tau=0.7)], 0, (1,) * 20),
             (cases.batch_problems(24, 7, 1e-2, 20, 120), 2, (1,) * 20),
             (cases.batch_problems(170, 7, 1e-2, 8, 40), 1, (70,))]

    def run(kind, out, start):
        probs, prec, calls = kind
        b = capi.Batch(probs, precision=prec)
        if start:
            start.wait()
        for n in calls:
            b.step(n)
        out.append(([b.f(k) for k in range(len(probs))], [b.stats(k) for k in range(len(probs))]))
        b.close()

    def serve(out, start):
        srv = capi.Server(5e8, max_slots=8, max_side=128, precision=2, lanes=2, split_side=64)
        if start:
            start.wait()
        ids = [srv.submit(cases.synthetic_problem(a, a + 7, 1e-2, seed=a, tau=0.5), 30) for a in (20, 40, 64, 100)]
        while srv.info()["completed"] < len(ids):
            srv.tick()
        got = [srv.poll(i) for i in ids]
        srv.close()
        out.append(([g[0] for g in got], [g[1] for g in got]))

    alone, mixed = [[] for _ in range(9)], [[] for _ in range(9)]
    for kind, out in zip(kinds, alone):
        run(kind, out, None)
    serve(alone[8], None)
    start = threading.Barrier(9)
    ts = [threading.Thread(target=run, args=(k, o, start)) for k, o in zip(kinds, mixed)]
    ts.append(threading.Thread(target=serve, args=(mixed[8], start)))
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, m in zip(alone, mixed):
        assert len(m) == 1
        _same(a[0], m[0])


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("ny", [1024, 1025])
def test_state_transposed_on_either_side(capi, ny, prec):
    """4096 cells go through the host, more through the device, in a batch whose instances are of both kinds:
    the states come back as they went in, to the other instances' none."""
    probs = [cases.synthetic_problem(a, b, 1e-2, seed=k, tau=0.7) for k, (a, b) in enumerate([(9, 7), (3, ny), (70, 66)])]
    b = capi.Batch(probs, precision=prec)
    before = [b.f(k) for k in range(3)]
    f = np.random.default_rng(ny).uniform(0.0, 1.0, (3, ny)) * 10.0 ** np.random.default_rng(1).uniform(-30, 30, (3, ny))
    b.set_f(1, f)
    got = [b.f(k) for k in range(3)]
    b.close()
    hi = f.astype(np.float32)
    want = f if prec == 0 else hi.astype(np.float64) + (f - hi).astype(np.float32).astype(np.float64)
    assert np.array_equal(got[1], want)
    assert np.array_equal(got[0], before[0]) and np.array_equal(got[2], before[2])


@pytest.mark.parametrize("prec", [0, 2])
@pytest.mark.parametrize("nx", [1439, 1440])
def test_dirichlet_values_at_the_last_launch(capi, nx, prec):
    """1440 values are the most that travel with launches; 1441 are copied."""
    test_dirichlet_values_of_any_number(capi, nx, prec)


@pytest.mark.parametrize("coop", [True, False])
@pytest.mark.parametrize("prec,tol", [(0, 1e-10), (1, 1e-8), (2, 1e-8)])
@pytest.mark.parametrize("precond", [0, 1])
def test_long_solves(capi, oracle, precond, prec, tol, coop):
    """A time step that leaves almost no diagonal: hundreds of iterations in one step, in FP64 in a single
    solve to the final tolerance, in which the residual's dot products only come from earlier sums."""
    p = cases.synthetic_problem(40, 36, 1e6, seed=11, tau=1e30)
    s = capi.Solver(p, precision=prec, precond=precond)
    s.set_coop(coop)
    s.update()
    f, st = s.f(), s.stats(0)
    s.close()
    ref = oracle.step(p, None, 1, solver="splu")
    assert st["status"] == capi.OK and st["iterations"] >= 150, st
    assert np.linalg.norm(f - ref) <= tol * np.linalg.norm(ref)
