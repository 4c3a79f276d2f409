"""Plain stream order (TURB_KV_PDL off) and kernels that start early give the
same bits: V-cycle, conjugate-gradient step, Helmholtz solves with immersed
rows, and the network of the learned guess, also when a context changes from
one to the other (its captured graphs hold the launches)."""
import numpy as np
import pytest

from tests import _cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guess", ["previous", "learned"])
@pytest.mark.parametrize("pmode", [0, 1])
def test_plain_order_is_bit_identical(pmode, guess):
    from turbins_gb300 import api as A
    from turbins_gb300 import build
    from turbins_gb300 import net as N
    build.build()
    case = _cases.bump_small(64, 32, 32)
    state = _cases.random_state(case, seed=3)
    plain, early = A.KV_ENO_SEGMENTS, A.KV_ENO_SEGMENTS | A.KV_PDL
    out = []
    for order in ((plain,) * 5, (early,) * 5, (early, early, plain, plain, early)):
        ctx = A.Context(case.grid, case.params)
        ctx.load_state(state)
        ctx.set_pressure_mode(pmode)
        net = None
        if guess == "learned":
            net = N.Net(64, 32, 32)
            net.init_params(2)
            N.set_learned_net(ctx, net)
            ctx.set_pressure_guess(A.GUESS_LEARNED)
            ctx.set_guess_galerkin(True)
        its = []
        for kv in order:   # the third and later steps have the history that a guess needs
            ctx.set_sweep_kernels(kv)
            st = ctx.step(case.dt)
            its.append((st["p_iters"], st["vel_iters"], st["conc_iters"]))
        out.append((its, ctx.pressure_guess_stats(), ctx.state()))
        ctx.close()
    for o in out[1:]:
        assert o[:2] == out[0][:2]
        for k in out[0][2]:
            assert np.array_equal(o[2][k], out[0][2][k]), k
    assert guess == "previous" or out[0][1][0] > 0
