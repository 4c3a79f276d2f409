"""The inner FP32 sweeps of the mixed Helmholtz solver follow the time step.

The sweeps of one defect correction are a captured graph that a context keeps.
A step with another dt has another 1/dt on the diagonal: a context that has
taken steps with other dt must take this one as a context that begins with it,
the same iteration counts and the same bits.  Where 1/dt makes up the diagonal
(here 64 to 1024 against about 1 of diffusion), sweeps that keep another
step's multiply the error by |1 - dt_kept / dt| per correction.
"""
import numpy as np
import pytest

from tests import _cases

pytestmark = pytest.mark.gpu

KEYS = ["u", "v", "w", "phi", "dpx", "dpy", "dpz", "c0"]


@pytest.mark.parametrize("inner", [2, 5])
@pytest.mark.parametrize("factors", [(1.0, 0.25, 4.0), (1.0, 0.5, 0.125, 2.0)])
def test_a_new_dt_reaches_the_inner_sweeps(factors, inner):
    from turbins_gb300 import api, build
    build.build()
    case = _cases.bump_small(24, 12, 8)

    def fresh(state):
        c = api.Context(case.grid, case.params)
        c.set_helmholtz_mode(api.HMODE_MIXED, inner)
        c.load_state(state)
        return c

    # powers of two: the kept diagonal, 1/dt_0 + (1/dt_1 - 1/dt_0) + .., is 1/dt exactly
    dt0 = 2.0 ** -8
    ctx = fresh(_cases.random_state(case, seed=5))
    for f in factors:
        before = {k: v for k, v in ctx.state().items() if k in KEYS}
        st = ctx.step(dt0 * f)
        other = fresh(before)
        so = other.step(dt0 * f)
        assert st["vel_iters"] == so["vel_iters"] and st["conc_iters"] == so["conc_iters"]
        got, want = ctx.state(), other.state()
        other.close()
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), (f, k)
    ctx.close()
