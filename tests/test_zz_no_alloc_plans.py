"""The scratch-free averaging's split by grid height: one row per block up to 592 rows, two up to 4096, four
up to the scratch array's 8192, against sums in extended precision; many calls in a row, which
wrap the counts of blocks; and values that are not finite.
"""
import ctypes

import numpy as np
import pytest

import effplast2d_b200 as ep

pytestmark = pytest.mark.gpu

FIELDS = ("P", "tauXX", "tauYY", "tauXY", "Ux", "Uy")


def _fields(nx, ny, seed):
    rng = np.random.default_rng(seed)
    dims = {"P": (ny, nx), "tauXX": (ny, nx), "tauYY": (ny, nx), "tauXY": (ny - 1, nx - 1), "Ux": (ny, nx + 1), "Uy": (ny + 1, nx)}
    f = {k: 1e-5 * rng.standard_normal(d) for k, d in dims.items()}
    f["P"] += 4e-5
    return f


def _expected(f, nx, ny, pa):
    """the eleven averages (EffPlast2D.cu:456-503) and a bound on their rounding errors: no term passes through more than
    256 additions (4 rows x 33 columns of a thread, a warp, 8 warps, 128 blocks of a lane, 16 lanes, and its own forming)"""
    L = np.longdouble
    g = {k: v.astype(L) for k, v in f.items()}
    dx, dy, nu0 = L(pa[0]), L(pa[1]), (1.5 * L(pa[3]) - L(pa[4])) / (3 * L(pa[3]) + L(pa[4]))
    px, py = int(nx / pa[10]), int(ny / pa[10])
    p, x, y, c = (g[k] for k in ("P", "tauXX", "tauYY", "tauXY"))
    zz, mzz = nu0 * (x + y - 2 * p), nu0 * (abs(x) + abs(y) + 2 * abs(p))
    a = np.s_[1:ny - 1, 1:nx - 1]
    j0, j1, i0, i1 = max(py + 1, 1), min(ny - py, ny - 1), max(px + 1, 1), min(nx - px, nx - 1)
    q = np.s_[j0:j1, i0:i1]
    at = lambda v, dj, di: v[j0 + dj:j1 + dj, i0 + di:i1 + di]
    ux, uy = g["Ux"], g["Uy"]
    ca = c[1:ny - 1, 1:nx - 1]
    cc = [at(c, -1, -1), at(c, -1, 0), at(c, 0, -1), at(c, 0, 0)]
    sx = [at(ux, 1, 0), at(ux, -1, 0), at(ux, 1, 1), at(ux, -1, 1)]  # + - + -, their differences telescope
    sy = [at(uy, 0, 1), at(uy, 0, -1), at(uy, 1, 1), at(uy, 1, -1)]
    alt = lambda v: v[0] - v[1] + v[2] - v[3]
    mag = lambda v: 2 * sum(abs(e) for e in v)
    all_, xy, inner = L(nx * ny), L((nx - 1) * (ny - 1)), L((nx - 2 * px) * (ny - 2 * py))
    terms = [(((x - p)[a]), (abs(x) + abs(p))[a], all_), ((y - p)[a], (abs(y) + abs(p))[a], all_),
             (ca + zz[a], abs(ca) + mzz[a], xy), (L(0) * ca, L(0) * ca, all_),
             ((x - p)[q], (abs(x) + abs(p))[q], inner), ((y - p)[q], (abs(y) + abs(p))[q], inner),
             (sum(cc) / 4, sum(abs(e) for e in cc) / 4, inner), (zz[q], mzz[q], inner),
             ((at(ux, 0, 1) - at(ux, 0, 0)) / dx, (abs(at(ux, 0, 1)) + abs(at(ux, 0, 0))) / dx, inner),
             ((at(uy, 1, 0) - at(uy, 0, 0)) / dy, (abs(at(uy, 1, 0)) + abs(at(uy, 0, 0))) / dy, inner),
             ((alt(sx) / dy + alt(sy) / dx) / 8, ((mag(sx) + 4 * abs(at(ux, 0, 0)) + 4 * abs(at(ux, 0, 1))) / dy +
                                                  (mag(sy) + 4 * abs(at(uy, 0, 0)) + 4 * abs(at(uy, 1, 0))) / dx) / 8, inner)]
    return [(float(t.sum() / d), float(m.sum() / abs(d)) * 256 * 2.0**-53) for t, m, d in terms]


def _call(dev, nx, ny, pa, out):
    rc = ep.lib().ep2d_average_fields_noalloc(nx, ny, (ctypes.c_double * 11)(*pa), *[ctypes.c_void_p(dev[f].data_ptr()) for f in FIELDS],
                                              ctypes.c_void_p(out.data_ptr()), None)
    assert rc == 0, ep.lib().ep2d_last_error()


@pytest.mark.parametrize("nx,ny", [(67, 593), (67, 594), (67, 595), (600, 597), (33, 4097), (33, 4098), (33, 4099), (35, 8193), (35, 8194)])
def test_averages_of_every_split(nx, ny):
    import torch

    pa = ep.make_pa(20.0, 20.0, nx, ny, porosity=0.01, n_pores=3)
    f = _fields(nx, ny, 90)
    dev = {k: torch.from_numpy(v).to("cuda") for k, v in f.items()}
    out = torch.full((11,), float("nan"), dtype=torch.float64, device="cuda")
    want = _expected(f, nx, ny, pa)
    first = None
    for call in range(3):
        out.fill_(float("nan"))
        _call(dev, nx, ny, pa, out)
        got = out.cpu().tolist()
        for k, (v, bound) in enumerate(want):
            assert abs(got[k] - v) <= bound, (call, k, got[k], v, bound)
        assert first in (None, got)
        first = got


def test_averages_of_many_calls():
    # more calls than there are counts of blocks, of two splits in turn
    import torch

    cases = []
    for nx, ny in ((67, 601), (64, 64)):
        pa = ep.make_pa(20.0, 20.0, nx, ny, porosity=0.01, n_pores=3)
        dev = {k: torch.from_numpy(v).to("cuda") for k, v in _fields(nx, ny, 91).items()}
        cases.append((dev, nx, ny, pa))
    outs = torch.full((600, 11), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for k in range(600):
        _call(*cases[k & 1], outs[k])
    torch.cuda.synchronize()
    assert torch.isfinite(outs).all()
    assert (outs[0::2] == outs[0]).all() and (outs[1::2] == outs[1]).all()


def test_averages_of_values_that_are_not_finite():
    # they reach the averages they are a term of, and no other
    import torch

    nx, ny = 70, 620
    pa = ep.make_pa(20.0, 20.0, nx, ny, porosity=0.01, n_pores=3)
    out = torch.zeros(11, dtype=torch.float64, device="cuda")
    f = _fields(nx, ny, 92)
    dev = {k: torch.from_numpy(v).to("cuda") for k, v in f.items()}
    _call(dev, nx, ny, pa, out)
    clean = out.cpu().numpy()
    for field, value, touched in (("P", np.nan, (0, 1, 2, 4, 5, 7)), ("tauXY", np.inf, (2, 6)), ("Ux", -np.inf, (8, 10)), ("Uy", np.nan, (9, 10))):
        dev = {k: torch.from_numpy(v).to("cuda") for k, v in f.items()}
        dev[field][300, 35] = value
        _call(dev, nx, ny, pa, out)
        got = out.cpu().numpy()
        for k in range(11):
            if k in touched:
                assert not np.isfinite(got[k]), (field, k)
            else:
                assert got[k] == clean[k], (field, k)
