"""Edges of the tiles, field groups and column segments of the step's kernels.

K1 and K2 give the same bits however a column is cut along k (whole, equal segments, single
levels, the default cut with its short segments), for every scheme in both forms, at field
counts that fill and do not fill a pass; the FP64 form also agrees with the oracle at ragged
sizes.  The vertical solve in shared memory gives the bits of the streaming one, which grouped
launches run.  The adjoint kernels pass the dot-product test at the edges of their tiles.
Both of a dot product's sides are sums of products with a relative error of a few hundred
roundings at most, so they agree to 1e-12 of the sum of the products' magnitudes.
"""
import numpy as np
import pytest

from fdd3260_b200 import Mimica, _lib, config
from fdd3260_b200 import ensemble as E
from fdd3260_b200.autograd import AdvectionFunction, FnContext
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12   # FP64 form against the oracle: the transforms' round-off

FORMS = {"fp64": _lib.MG_PREC_FP64, "mixed": _lib.MG_PREC_MIXED}


def _fields(s):
    return [s.u, s.v, s.w, s.p, s.dens, *s.scal]


def _interior(a):
    return a[:, 3:-2, 3:-2]


def _run(d, st, cut):
    with Mimica(d, nscal=len(st.scal), iqt=1) as m:
        m.tune_set({**m.tune_get(), "k1_segments": cut[0], "k2_segments": cut[1]})
        m.upload(st)
        m.stepping(2, ntime0=1)
        return m.download()


# the last grid's default cut has short segments in both kernels
@pytest.mark.parametrize("maxx,maxy,nz,extra", [(8, 8, 8, 0), (36, 20, 11, 1), (40, 24, 30, 4), (160, 80, 36, 2)])
@pytest.mark.parametrize("scheme", ["weno", "ppm", "muscl", "lw", "quick"])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_column_cuts(form, scheme, maxx, maxy, nz, extra):
    d = config.cumulus_domain(maxx, maxy, nz, scheme=scheme, precision=FORMS[form])
    st = config.cumulus_state(d, seed=77, n_extra=extra)
    whole = _run(d, st, (1, 1))
    assert all(np.isfinite(a).all() for a in _fields(whole))
    for cut in [(0, 0), (3, 2), (nz, nz)]:
        for a, b in zip(_fields(_run(d, st, cut)), _fields(whole)):
            assert np.array_equal(a, b), cut
    if form == "fp64" and nz <= 11:
        r, _, _ = O.Oracle(d).stepping(st, nsteps=2, ntime0=1)
        for a, b in zip(_fields(whole), _fields(r)):
            assert np.abs(_interior(a) - _interior(b)).max() <= TOL * max(np.abs(_interior(b)).max(), 1e-300)


# groups of 8 levels; 302 levels are the most whose columns fit one CTA's shared memory
@pytest.mark.parametrize("nz", [8, 9, 33, 302, 303])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_vertical_solve_paths(form, nz):
    probs = [E.member_problem(E.MemberSpec(q, n, nz, 31 + q, 2.0, (n * 25.0, n * 25.0, 200.0)), precision=FORMS[form])
             for q, n in enumerate([16, 40])]
    alone = []
    for d, st in probs:
        with Mimica(d, nscal=len(st.scal), iqt=st.iqt) as m:
            m.upload(st)
            m.stepping(2, ntime0=1)
            alone.append(m.download())
    members = [Mimica(d, nscal=len(st.scal), iqt=st.iqt) for d, st in probs]
    try:
        for m, (d, st) in zip(members, probs):
            m.upload(st)
        with E.Ensemble(members, mode="grouped") as ens:
            ens.step(2, ntime0=1)
        for m, a in zip(members, alone):
            for x, y in zip(_fields(a), _fields(m.download())):
                assert np.isfinite(x).all() and np.array_equal(x, y)
    finally:
        for m in members:
            m.close()


def _advected(d, seed):
    rng = np.random.default_rng(seed)
    st = config.random_state(d, seed=seed)
    mom = [st.u * d.den0[:, None, None], st.v * d.den0[:, None, None], st.w * d.avden0[:, None, None]]
    mom[2][0] = 0.0

    def field(scale, periodic=True):
        a = np.zeros(d.shape)
        a[:, 3:-2, 3:-2] = scale * rng.standard_normal(_interior(a).shape)
        return config.periodic_fill(a) if periodic else a

    return st, [config.periodic_fill(a) for a in mom], field


# tiles of 61 (x) and 29 (y, z) cells over the cells with their ghosts: less than one, one tile exactly (y, z), one and
# a remainder
@pytest.mark.parametrize("maxx,maxy,nz", [(8, 8, 8), (54, 24, 29), (64, 30, 32)])
def test_scalar_adjoint_tiles(maxx, maxy, nz):
    d = config.cumulus_domain(maxx, maxy, nz)
    st, mom, field = _advected(d, 5)
    dx, dm = field(1.0), [field(0.1), field(0.1), field(0.05)]
    dm[2][0] = 0.0
    abar = field(1.0, periodic=False)
    with Mimica(d, nscal=2) as m:
        ctx = FnContext(m)
        AdvectionFunction.forward(ctx, st.scal[0] * st.dens, *mom)
        tl = AdvectionFunction.jvp(ctx, dx, *dm)
        bars = AdvectionFunction.backward(ctx, abar)
    rhs = sum(float(np.sum(a * b)) for a, b in zip([dx, *dm], bars))
    assert abs(float(np.sum(tl * abar)) - rhs) <= 1e-12 * float(np.sum(np.abs(tl * abar)))


# levels 5 .. nz-4 take the instance without level tests: none of 8 levels, one of 9, 4 of 12
@pytest.mark.parametrize("maxx,nz", [(16, 8), (16, 9), (144, 12)])
@pytest.mark.parametrize("mom_ord", [4, 2])
def test_momentum_adjoint_levels(mom_ord, maxx, nz):
    d = config.cumulus_domain(maxx, 16, nz, mom_ord=mom_ord)
    st, mom, field = _advected(d, 6)
    dm = [field(1.0), field(1.0), field(0.5)]
    lam = [field(1.0, periodic=False) for _ in range(3)]
    with Mimica(d, nscal=1) as m:
        tl = m.qnadv_tl(*mom, *dm, 1)
        ad = m.qnadv_ad(*mom, *lam, 1)
    gross = sum(float(np.sum(np.abs(_interior(t) * _interior(q)))) for t, q in zip(tl, lam))
    lhs = sum(float(np.sum(_interior(t) * _interior(q))) for t, q in zip(tl, lam))
    rhs = sum(float(np.sum(_interior(x) * _interior(a))) for x, a in zip(dm, ad))
    assert abs(lhs - rhs) <= 1e-12 * gross
