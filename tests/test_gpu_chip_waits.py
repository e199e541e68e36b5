"""The on-chip form's bounded waits and the turns of handles that share a device.

Nothing here faults: CTAs are left out of a launch, the others' waits run out after a few
milliseconds, the launch ends, and the context stays usable.
"""
import numpy as np
import pytest

import effplast2d_b200 as ep
from test_gpu_chip import _run
from test_gpu_kernels import FIELDS, _pa, _random_state

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
