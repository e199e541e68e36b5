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
