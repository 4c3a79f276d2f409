"""Helmholtz solves of one context in changing forms.

An FP64 solve exchanges the solution's array with a spare one, and the mixed
solver's captured sweeps add their correction to the array they were captured
with: a context that changes between the modes, or the number of inner sweeps
(with one there is no captured sweep at all), must step as a context that
begins with that form, the same iteration counts and the same bits.
"""
import numpy as np
import pytest

from tests import _cases

pytestmark = pytest.mark.gpu

KEYS = ["u", "v", "w", "phi", "dpx", "dpy", "dpz", "c0"]
FP64, MIXED = 0, 1


def _fresh(api, case, state, mode, inner):
    c = api.Context(case.grid, case.params)
    c.set_helmholtz_mode(mode, inner)
    c.load_state(state)
    return c


@pytest.mark.parametrize("forms", [[(MIXED, 5), (FP64, 5), (MIXED, 5), (FP64, 5), (FP64, 5), (MIXED, 5)],
                                   [(FP64, 1), (MIXED, 3), (FP64, 1), (MIXED, 3)],
                                   [(MIXED, 5), (MIXED, 1), (MIXED, 2), (MIXED, 1), (MIXED, 5), (MIXED, 6)]])
def test_a_context_may_change_its_helmholtz_form(forms):
    from turbins_gb300 import api, build
    build.build()
    case = _cases.bump_small(24, 12, 8)
    ctx = api.Context(case.grid, case.params)
    ctx.load_state(_cases.random_state(case, seed=9))
    for mode, inner in forms:
        before = {k: v for k, v in ctx.state().items() if k in KEYS}
        ctx.set_helmholtz_mode(mode, inner)
        st = ctx.step(case.dt)
        other = _fresh(api, case, before, mode, inner)
        so = other.step(case.dt)
        assert st["vel_iters"] == so["vel_iters"] and st["conc_iters"] == so["conc_iters"], (mode, inner)
        got, want = ctx.state(), other.state()
        other.close()
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), (mode, inner, k)
    ctx.close()


@pytest.mark.parametrize("inner", [1, 2])
@pytest.mark.parametrize("mk", [lambda: _cases.bump_small(), lambda: _cases.multi_small()])
def test_few_inner_sweeps_solve(mk, inner):
    """one sweep per correction (the residual's own, added by k_add_corr) and
    two (the last one alone): the operator applied to the solution leaves the
    residual the solve promises, |b - A x| <= vel_rtol |b|, but for the rounding
    of some ten FP64 operations per row in either evaluation"""
    from turbins_gb300 import api, build
    build.build()
    case = mk()
    s = _cases.random_state(case, seed=13)
    dt = case.dt
    ctx = _fresh(api, case, s, MIXED, inner)
    for q, f, fb in (("u", api.F_U, api.F_B_U), ("v", api.F_V, api.F_B_V), ("w", api.F_W, api.F_B_W)):
        b = s[q] / dt + 0.1
        b[case.grid.status[q] != 3] = 0.0
        ctx.upload(fb, b)
        assert ctx.Velocity_solve(q, dt) > 0
        ctx.helmholtz_apply(q, 0, dt, f, api.F_SCRATCH0)
        r = b - ctx.download(api.F_SCRATCH0)
        assert np.linalg.norm(r) <= (case.params.vel_rtol + 1e-14) * np.linalg.norm(b)
    ctx.close()
