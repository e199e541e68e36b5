"""The on-chip form's bounded waits and the turns of handles that share a device.

Nothing here faults: CTAs are left out of a launch, the others' waits run out after a few
milliseconds, the launch ends, and the context stays usable.
"""
import threading
import time

import numpy as np
import pytest

import effplast2d_b200 as ep
from effplast2d_b200 import batch as B
from test_gpu_chip import _run
from test_gpu_kernels import FIELDS, PLASTIC_FIELDS, _pa, _random_state

pytestmark = pytest.mark.gpu


def _solver(nx, ny, seed=80, **kw):
    kw = dict(dict(nl=2), **kw)
    s = ep.Solver(nx, ny, _pa(nx, ny, n_pores=2, porosity=0.03, yield_stress=1e-5), **kw)
    return s, _random_state(nx, ny, seed)


def _set(s, st):
    for k, v in st.items():
        s.set(k, v)


@pytest.mark.parametrize("nx,ny", [(64, 64), (301, 203), (1024, 1024)])
def test_wait_for_a_missing_neighbour_runs_out(nx, ny):
    s, st = _solver(nx, ny)
    _set(s, st)
    s.check_chip_wait(missing=1)
    for _ in range(2):  # the second launch finds the flag set and returns at once
        with pytest.raises(ep.EP2DError) as e:
            s.iterate(40)
        assert e.value.status == ep.ERR_CUDA and "ran out" in str(e.value)
    s.close()
    pa = _pa(nx, ny, n_pores=2, porosity=0.03, yield_stress=1e-5)
    a, _ = _run(nx, ny, pa, 2, st, (40,), ep.FP64, kernel=ep.KERNEL_STREAM, rows=16)
    b, _ = _run(nx, ny, pa, 2, st, (40,), ep.FP64)
    for f in FIELDS:
        assert np.array_equal(a[f], b[f]), f


def test_chip_wait_arguments():
    s, _ = _solver(16, 16)
    for kw in (dict(missing=-1), dict(missing=1, timeout_ns=-1), dict(missing=1, timeout_ns=20_000_000_000)):
        with pytest.raises(ep.EP2DError) as e:
            s.check_chip_wait(**kw)
        assert e.value.status == ep.ERR_ARG
    s.close()


@pytest.mark.parametrize("precision", [ep.FP64, ep.F32_BULK], ids=["fp64", "f32"])
def test_reset_after_a_failed_wait_gives_a_fresh_handle(precision):
    # (in the FP32 phase the failed step also leaves the state in its FP32 form)
    nx, ny = 130, 96
    kw = dict(niter=120, check_every=40, precision=precision)
    s, _ = _solver(nx, ny, **kw)
    s.check_chip_wait(missing=1)
    with pytest.raises(ep.EP2DError) as e:
        s.solve_step(0, -6e-5, [1.0, 0.8, 0.3])
    assert e.value.status == ep.ERR_CUDA
    s.reset()
    r = s.solve_step(0, -6e-5, [1.0, 0.8, 0.3])[0]
    t, _ = _solver(nx, ny, **kw)
    q = t.solve_step(0, -6e-5, [1.0, 0.8, 0.3])[0]
    assert r["iterations"] == q["iterations"] and r["sigma"] == q["sigma"]
    for f in FIELDS:
        assert np.array_equal(s.get(f), t.get(f)), f
    s.close()
    t.close()


# 2047 x 64 has 74 tiles beside one another: those far from the missing ones have gone through the 9
# iterations of the first launch when it gives up
@pytest.mark.parametrize("nx,ny", [(64, 64), (301, 203), (2047, 64), (1024, 1024)])
@pytest.mark.parametrize("nl,precision", [(1, ep.FP64), (3, ep.FP64), (2, ep.MIXED)], ids=["elastic", "plastic", "mixed"])
def test_launch_whose_ctas_cannot_all_start(nx, ny, nl, precision):
    pa = _pa(nx, ny, n_pores=2, porosity=0.03, yield_stress=1e-5)
    st = _random_state(nx, ny, 81)
    out = []
    for missing in (0, 1, 3):
        s = ep.Solver(nx, ny, pa, nl=nl, precision=precision)
        _set(s, st)
        if missing:
            s.check_chip_start(missing)
        for n in (10, 33, 1):
            s.iterate(n)
        out.append({f: s.get(f) for f in FIELDS + PLASTIC_FIELDS})
        if missing:  # the plain iterations after the first attempt were single launches
            assert s.stats()["launches"] > 20
        s.close()
    for o in out[1:]:
        for f in o:
            assert np.array_equal(o[f], out[0][f]), f


@pytest.mark.parametrize("precision", [ep.FP64, ep.MIXED, ep.F32_BULK], ids=["fp64", "mixed", "f32"])
@pytest.mark.parametrize("niter", [120, 100], ids=["checkpoint-last", "no-checkpoint-last"])
def test_solve_goes_on_when_ctas_cannot_start(precision, niter):
    # with the plastic zone tracked; the interval that gives up is the first, with the recording
    # launch behind it, or (second step of a handle) the FP32 phase's
    nx, ny = 130, 96
    out = []
    for missing in (0, 2):
        s, _ = _solver(nx, ny, niter=niter, check_every=40, precision=precision)
        s.track_plastic_zone(True)
        if missing:
            s.check_chip_start(missing)
        r = s.solve_step(0, -6e-5, [1.0, 0.8, 0.3], 2)
        p = s.polar_fields(-6e-5)
        out.append(([(q["iterations"], q["sigma"], q["error"]) for q in r], s.check_errors(0, 0), p,
                    {f: s.get(f) for f in FIELDS}))
        s.close()
    assert out[0][0] == out[1][0] and out[0][1] == out[1][1]
    for k in (2, 3):
        for f in out[0][k]:
            assert np.array_equal(out[0][k][f], out[1][k][f]), f


@pytest.mark.parametrize("precision", [ep.FP64, ep.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("missing", [1, 100])
def test_batch_goes_on_when_ctas_cannot_start(precision, missing):
    # of the RVEs of one launch some have their CTAs and some not
    specs = []
    for k, n in enumerate([512, 300, 310]):
        pa = ep.make_pa(20.0, 20.0, n, n, yield_stress=1e-5, porosity=0.01, n_pores=1)
        specs.append(B.spec(n, pa, 1 + k % 3, 1, -6e-5, (1.0, 0.8, 0.3)))
    kw = dict(niter=160, check_every=80, precision=precision)
    a, sa = B.batch_solve(specs, **kw)
    b, sb = B.batch_solve(specs, check_start=(missing, 2_000_000), **kw)
    assert sb["launches"] > sa["launches"] + 100
    for x, y in zip(a, b):
        assert x["total_iterations"] == y["total_iterations"]
        for m in ("kphi", "kd", "g"):
            u, v = x["num"][m], y["num"][m]
            assert u == v or (np.isnan(u) and np.isnan(v)), (m, u, v)


def test_check_start_arguments():
    s, _ = _solver(16, 16)
    for kw in (dict(missing=-1), dict(missing=1, timeout_ns=-1), dict(missing=1, timeout_ns=20_000_000_000)):
        with pytest.raises(ep.EP2DError) as e:
            s.check_chip_start(**kw)
        assert e.value.status == ep.ERR_ARG
    s.close()


@pytest.mark.parametrize("room", [0, 1, 2])
def test_batch_goes_on_when_the_device_refuses_a_wave(room):
    # the two waves of the first interval and the one of the second: each refused in turn
    specs = []
    for k, n in enumerate([700, 640, 512, 300, 33]):
        pa = ep.make_pa(20.0, 20.0, n, n, yield_stress=1e-5, porosity=0.01, n_pores=1)
        specs.append(B.spec(n, pa, 1 + k % 2, 1, -6e-5, (1.0, 0.8, 0.3)))
    kw = dict(niter=161, check_every=161)
    a, sa = B.batch_solve(specs, **kw)
    b, sb = B.batch_solve(specs, check_room=room, **kw)
    assert sa["launches"] < 20 and sb["launches"] > sa["launches"] + 100
    for x, y in zip(a, b):
        assert x["total_iterations"] == y["total_iterations"]
        for m in ("kphi", "kd", "g"):
            u, v = x["num"][m], y["num"][m]
            assert u == v or (np.isnan(u) and np.isnan(v)), (m, u, v)


def _in_threads(work, args):
    bar = threading.Barrier(len(args) + 1)

    def run(a):
        bar.wait()
        work(*a)

    ths = [threading.Thread(target=run, args=(a,)) for a in args]
    for t in ths:
        t.start()
    bar.wait()
    t0 = time.perf_counter()
    for t in ths:
        t.join()
    return time.perf_counter() - t0


def test_small_handles_run_side_by_side():
    # eight 128^2 handles in eight threads: one after another they would take eight times one
    # handle's time (a quarter of that was measured with shares of the SMs)
    n = 128
    hs = [_solver(n, n, nl=3, niter=8000, eiter=0.0, check_every=2000)[0] for _ in range(8)]

    def solve(h):
        h.solve_step(0, -6e-5, [1.0, 0.8, 0.3])

    for h in hs:
        solve(h)
    one = min(_in_threads(solve, [(hs[0],)]) for _ in range(3))
    all_ = min(_in_threads(solve, [(h,) for h in hs]) for _ in range(3))
    assert all_ < 0.7 * 8 * one, (all_, one)
    for h in hs:
        h.close()


def test_handles_of_all_kinds_side_by_side():
    # shapes for any share of the SMs, beside a batch: each result as alone
    kinds = [(48, 64, dict(nl=1)), (64, 64, dict(nl=3)), (128, 130, dict(nl=3)), (200, 90, dict(nl=2, precision=ep.MIXED)),
             (301, 203, dict(nl=2, track=True)), (256, 256, dict(nl=2, precision=ep.F32_BULK)), (512, 500, dict(nl=3)),
             (640, 640, dict(nl=1)), (1024, 1024, dict(nl=2)), (128, 128, dict(nl=1, kernel=ep.KERNEL_RESIDENT, rows=8))]
    specs = [B.spec(n, ep.make_pa(20.0, 20.0, n, n, yield_stress=1e-5, porosity=0.01, n_pores=1), 2, 1, -6e-5, (1.0, 0.8, 0.3))
             for n in (700, 640, 512, 300, 64)]

    def handle(nx, ny, kw):
        kw = dict(kw)
        track = kw.pop("track", False)
        s, _ = _solver(nx, ny, niter=1600, eiter=0.0, check_every=200, **kw)
        if track:
            s.track_plastic_zone(True)
        r = s.solve_step(0, -6e-5, [1.0, 0.8, 0.3])[0]
        out = {f: s.get(f) for f in FIELDS}
        if track:
            out.update(s.polar_fields(-6e-5))
        s.close()
        return r["sigma"], out

    def batch():
        return [[r["num"][m] for m in ("kphi", "kd", "g")] for r in B.batch_solve(specs, niter=800, check_every=400, eiter=0.0)[0]]

    want, want_b = [handle(*k) for k in kinds], batch()
    got, got_b = [None] * len(kinds), [None]

    def work(k):
        if k < len(kinds):
            got[k] = handle(*kinds[k])
        else:
            got_b[0] = batch()

    _in_threads(work, [(k,) for k in range(len(kinds) + 1)])
    assert np.array_equal(np.array(got_b[0]), np.array(want_b), equal_nan=True)
    for k, (sigma, fields) in enumerate(want):
        assert got[k][0] == sigma, kinds[k]
        for f in fields:
            assert np.array_equal(got[k][1][f], fields[f]), (kinds[k], f)
