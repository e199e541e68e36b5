"""The on-chip form: a run of plain iterations in one launch, the state on the SMs.

The library takes it (kernel AUTO) for runs of 8 plain iterations or more on grids that fit on chip.
It evaluates the same per-cell formulas as the other forms, so every field must
equal the stream form's bit for bit.  The grids sit at the edges of its split: one tile,
one column or row past a 28-column strip or a tile of rows, the widest and tallest that
fit at a given number of rows per warp (2 to 18), and the first that does not fit.
"""
import threading

import numpy as np
import pytest

import effplast2d_b200 as ep
from effplast2d_b200 import batch as B
from test_gpu_kernels import FIELDS, PLASTIC_FIELDS, _pa, _random_state

pytestmark = pytest.mark.gpu


def _run(nx, ny, pa, nl, st, counts, precision, **kw):
    s = ep.Solver(nx, ny, pa, nl=nl, precision=precision, **kw)
    for k, v in st.items():
        s.set(k, v)
    for n in counts:
        s.iterate(n)
    out = {f: s.get(f) for f in FIELDS + PLASTIC_FIELDS}  # (elastic: the latter stay zero)
    launches = s.stats()["launches"]
    s.close()
    return out, launches


# (8, 8): one tile, smaller than it in both directions; 28, 29, 57: strips of 28 columns and
# one column over; rows 2 to 18 per warp (chip_shape: 128^2 2, 400^2 4, 520^2 6, 700^2 10, 1024^2 16,
# 1060^2 18); 1100^2 does not fit and stays with the stream form
GRIDS = [(8, 8), (28, 17), (29, 9), (57, 130), (128, 128), (301, 203), (403, 401), (521, 517), (64, 2047), (2047, 64),
         (700, 699), (1024, 1024), (1061, 1060), (1100, 1100)]


@pytest.mark.parametrize("nx,ny", GRIDS, ids=["%dx%d" % g for g in GRIDS])
@pytest.mark.parametrize("nl,precision", [(1, ep.FP64), (3, ep.FP64), (2, ep.MIXED)], ids=["elastic", "plastic", "mixed"])
def test_chip_form_matches_stream_form(nx, ny, nl, precision):
    pa = _pa(nx, ny, n_pores=2, porosity=0.03, yield_stress=1e-5)
    st = _random_state(nx, ny, 41)
    counts = (9, 1, 30, 33)  # runs of 8, 29 and 32 plain iterations: both parities
    a, la = _run(nx, ny, pa, nl, st, counts, precision, kernel=ep.KERNEL_STREAM, rows=16)
    b, lb = _run(nx, ny, pa, nl, st, counts, precision)
    for f in a:
        assert np.array_equal(b[f], a[f], equal_nan=True), (f, float(np.nanmax(np.abs(b[f] - a[f]))))
    assert la == 73
    if max(nx, ny) < 1100 or min(nx, ny) == 64:
        assert lb == 7  # three on-chip launches, four recording ones


@pytest.mark.parametrize("nx,ny", [(9, 12), (96, 131), (257, 256), (530, 300), (1061, 1060)])
@pytest.mark.parametrize("precision", [ep.FP64, ep.MIXED], ids=["fp64", "mixed"])
def test_chip_tracking_matches_stream_tracking(nx, ny, precision):
    # the yield bits of every iteration, single launches and on-chip runs alike, and the fields
    pa = _pa(nx, ny, n_pores=1, porosity=0.02, yield_stress=1e-5)
    st = _random_state(nx, ny, 61)
    out = []
    for kw in (dict(kernel=ep.KERNEL_STREAM, rows=16), {}):
        s = ep.Solver(nx, ny, pa, nl=2, precision=precision, **kw)
        for k, v in st.items():
            s.set(k, v)
        s.track_plastic_zone(True)
        s.iterate(40)
        s.iterate(3)
        s.iterate(61)
        d = s.polar_fields(-6e-5)
        d.update({f: s.get(f) for f in ("Ux", "Vy", "J2XY")})
        out.append(d)
        s.close()
    assert out[0]["Plast"].max() > 0
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("rows", [4, 5, 19, 37, 200])
@pytest.mark.parametrize("nl,precision", [(1, ep.FP64), (3, ep.FP64), (2, ep.MIXED)], ids=["elastic", "plastic", "mixed"])
def test_stream_pairs_match_tile_form(rows, nl, precision):
    # the stream form's plain launches march two rows per step: odd and even segments, the last
    # one cut short, interior and edge segments, a ragged last strip
    nx, ny = 203, 181
    pa = _pa(nx, ny, n_pores=3, porosity=0.03, yield_stress=1e-5)
    st = _random_state(nx, ny, 43)
    a, _ = _run(nx, ny, pa, nl, st, (70, 2), precision, kernel=ep.KERNEL_TILE, rows=16)
    b, _ = _run(nx, ny, pa, nl, st, (70, 2), precision, kernel=ep.KERNEL_STREAM, rows=rows)
    for f in a:
        assert np.array_equal(b[f], a[f]), (f, float(np.max(np.abs(b[f] - a[f]))))


# states above PAIR_TURN_BYTES, whose marches go up and down in turn: the library's segments and odd
# and even ones, tall and wide grids of a ragged last strip and segment
@pytest.mark.parametrize("nx,ny,rows", [(1801, 1699, 0), (203, 15001, 37), (15001, 201, 6)])
@pytest.mark.parametrize("nl,precision", [(1, ep.FP64), (3, ep.FP64), (2, ep.MIXED)], ids=["elastic", "plastic", "mixed"])
def test_marches_in_turn_match_tile_form(nx, ny, rows, nl, precision):
    pa = _pa(nx, ny, n_pores=3, porosity=0.03, yield_stress=1e-5)
    st = _random_state(nx, ny, 47)
    rng = np.random.default_rng(48)
    st["Vy"][0] = 1e-7 * rng.standard_normal(nx)  # row 0 of Uy moves with its velocity, row ny never does
    st["Vy"][-1] = 1e-7 * rng.standard_normal(nx)
    form = dict(kernel=ep.KERNEL_STREAM, rows=rows) if rows else {}
    a, _ = _run(nx, ny, pa, nl, st, (8, 3), precision, kernel=ep.KERNEL_TILE, rows=16)
    b, _ = _run(nx, ny, pa, nl, st, (8, 3), precision, **form)
    for f in a:
        assert np.array_equal(b[f], a[f]), (f, float(np.max(np.abs(b[f] - a[f]))))


def test_marches_in_turn_f32():
    # FP32: the same iterations from either buffer, so each is once a march up and once a march down
    nx, ny = 2400, 2003
    pa = _pa(nx, ny, n_pores=3, porosity=0.03, yield_stress=1e-5)
    st = _random_state(nx, ny, 49)
    out = []
    for first in (0, 1):
        s = ep.Solver(nx, ny, pa, nl=2, precision=ep.F32_BULK)
        s.iterate_f32(first)
        for k, v in st.items():
            s.set(k, v)
        s.iterate_f32(5)
        out.append({f: s.get(f) for f in ("Ux", "Uy", "Vx", "Vy")})
        s.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f
        assert not np.array_equal(out[0][f], st[f])


@pytest.mark.parametrize("nx,ny", [(8, 9), (57, 130), (403, 401), (1061, 1060)])
@pytest.mark.parametrize("nl", [1, 2])
def test_chip_f32_matches_stream_f32(nx, ny, nl):
    # the FP32 bulk's iterations on chip against single launches of the stream form; the
    # recorded stresses are left alone
    pa = _pa(nx, ny, n_pores=1, porosity=0.02, yield_stress=1e-5)
    out = []
    for kw in (dict(kernel=ep.KERNEL_STREAM, rows=16), {}):
        s = ep.Solver(nx, ny, pa, nl=nl, niter=40, check_every=40, precision=ep.F32_BULK, **kw)
        s.solve_step(0, -6e-5, [1.0, 0.8, 0.3])
        p = s.get("P")
        for n in (41, 30):
            s.iterate_f32(n)
        assert np.array_equal(s.get("P"), p)
        out.append({f: s.get(f) for f in ("Ux", "Uy", "Vx", "Vy")})
        s.close()
    for f in out[0]:
        assert np.max(np.abs(out[0][f])) > 0.0
        assert np.array_equal(out[0][f], out[1][f]), f


def test_chip_form_two_threads():
    # on-chip launches of different handles take turns; both finish with the single-thread result
    nx = ny = 200
    pa = _pa(nx, ny, n_pores=3, porosity=0.02, yield_stress=1e-5)
    sts = [_random_state(nx, ny, 50 + k) for k in range(2)]
    want = [_run(nx, ny, pa, 3, st, (400,), ep.FP64)[0] for st in sts]
    got = [None, None]

    def work(k):
        got[k] = _run(nx, ny, pa, 3, sts[k], (100,) * 4, ep.FP64)[0]

    ths = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ths:
        t.start()
    for t in ths:
        t.join()
    for k in range(2):
        for f in ("Ux", "Uy", "Vx", "Vy"):
            assert np.array_equal(got[k][f], want[k][f]), (k, f)


@pytest.mark.parametrize("precision", [ep.FP64, ep.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sides", [[8 + 3 * (k % 20) for k in range(70)], [700, 640, 512, 300, 33]],
                         ids=["more-than-a-launch-takes", "two-waves"])
def test_batch_waves_match_stream_batch(sides, precision):
    # on-chip waves (AUTO) against the batched stream launches (pinned shape), elastic and
    # plastic RVEs side by side: equal results
    specs = []
    for k, n in enumerate(sides):
        pa = ep.make_pa(20.0, 20.0, n, n, yield_stress=1e-5, porosity=0.005 + 0.0005 * (k % 7), n_pores=1)
        specs.append(B.spec(n, pa, 1 + k % 3, 1, -6e-5, (1.0, 0.8, 0.3)))
    kw = dict(niter=800, check_every=400, precision=precision)
    a, _ = B.batch_solve(specs, kernel=ep.KERNEL_STREAM, rows=16, **kw)
    b, _ = B.batch_solve(specs, **kw)
    for x, y in zip(a, b):
        assert x["total_iterations"] == y["total_iterations"]
        for kind in ("num", "num_per", "an"):
            for m in ("kphi", "kd", "g"):
                u, v = x[kind][m], y[kind][m]
                assert u == v or (np.isnan(u) and np.isnan(v)), (kind, m, u, v)


@pytest.mark.parametrize("kw,n", [(dict(kernel=ep.KERNEL_STREAM, rows=16), 1200), (dict(kernel=ep.KERNEL_RESIDENT, rows=8), 160)],
                         ids=["stream", "resident"])
def test_chip_form_beside_another_handle(kw, n):
    # a small grid's CTAs (few warps, little shared memory) find their SMs while another thread's
    # launches come and go, or another form's CTAs wait on one another; both results as alone
    cases = [(64, {}, (500,) * 6), (n, kw, (300,) * 3)]
    ins = [(m, m, _pa(m, m, n_pores=3, porosity=0.02, yield_stress=1e-5), 3, _random_state(m, m, 70), counts, ep.FP64, k)
           for m, k, counts in cases]
    want = [_run(*a, **k)[0] for *a, k in ins]
    got = [None, None]

    def work(k):
        *a, opt = ins[k]
        got[k] = _run(*a, **opt)[0]

    ths = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ths:
        t.start()
    for t in ths:
        t.join()
    for k in range(2):
        for f in ("Ux", "Uy", "Vx", "Vy"):
            assert np.array_equal(got[k][f], want[k][f]), (k, f)
