"""ENO convection where its forms of one operation could part from the plain
one: every order on uniform power-of-two, uniform other and stretched
spacings, node counts around the segment lengths, and fields whose values
run from subnormal to 1e140, with zeros of both signs (exact scalings, halved
interpolation weights and fused products are only taken where they round as
the plain operations).  Compared bit for bit with the oracle and with the IEEE
division mode."""
import numpy as np
import pytest

from tests import _cases
from turbins_gb300 import workload as W

pytestmark = pytest.mark.gpu

# cells, lengths, y stretching: spacings of the axes that are powers of two
BOXES = {"pow2": ((32, 16, 16), (8.0, 1.0, 1.0), None), "other": ((20, 12, 12), (3.0, 1.0, 0.7), None),
         "stretched": ((12, 36, 8), (3.0, 1.0, 0.5), 1.5), "long": ((8, 8, 72), (1.0, 1.0, 9.0), 1.2)}


def wide(case, seed):
    """velocities and concentrations over the whole exponent range"""
    rng = np.random.Generator(np.random.PCG64(seed))
    s = _cases.random_state(case, seed=seed)
    for k in ("u", "v", "w", "c0"):
        a = rng.standard_normal(case.grid.shape)
        e = rng.choice([0.0, -2.0, -100.0, -240.0, -300.0, -308.0, -318.0, 140.0], size=a.shape,
                       p=[0.5, 0.1, 0.05, 0.05, 0.1, 0.08, 0.07, 0.05])
        # runs of one magnitude, so that some stencils see only tiny values
        e = np.repeat(e[..., ::4], 4, axis=2)[..., :a.shape[2]]
        with np.errstate(under="ignore"):
            a = a * 10.0 ** e
        a[rng.random(a.shape) < 0.1] = 0.0
        a[rng.random(a.shape) < 0.05] = -0.0
        a[case.grid.status["c" if k == "c0" else k] == W.BOUNDARY] = 0.0
        s[k] = a
    return s


@pytest.mark.parametrize("values", ["plain", "wide"])
@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("box", sorted(BOXES))
def test_convection_forms(oracle_mod, box, order, values):
    from turbins_gb300 import api, build
    build.build()
    n, lengths, q = BOXES[box]
    case = W.poisson_case(*n, lengths, q)
    case.params.eno_order = order
    s = _cases.random_state(case, seed=order) if values == "plain" else wide(case, order)
    ctx = api.Context(case.grid, case.params)
    ctx.load_state(s)
    orc = oracle_mod.Oracle(case.grid, case.params)
    got = {}
    for fast in (1, 0):
        ctx.set_eno_division(fast)
        ctx.Velocity_cell_center()
        for f in "uvw":
            ctx.Velocity_convective_terms(f)
        ctx.Conc_convective_terms(0)
        got[fast] = [ctx.download(api.F_CONV_U + t) for t in range(3)] + [ctx.download(api.F_CCONV0)]
    ctx.close()
    tr = {f: orc.transpose(f, s["u"], s["v"], s["w"]) for f in "uvw"}
    adv = {"u": (s["u"],) + tuple(tr["u"]), "v": (tr["v"][0], s["v"], tr["v"][1]), "w": tuple(tr["w"]) + (s["w"],)}
    ref = [orc.convection_vel(f, s[f], *adv[f]) for f in "uvw"]
    ub, vb, wb = orc.cell_center(s["u"], s["v"], s["w"])
    ref.append(orc.convection_conc(0, s["c0"], ub, vb, wb))
    for a, b, r in zip(got[1], got[0], ref):
        assert np.array_equal(a, b, equal_nan=True)
        assert np.array_equal(a, r, equal_nan=True)
