"""The shared-memory cluster V-cycle of the lower levels (k_vcycle_low)
against a launch per half sweep: every cell's operations are the same, so the
Poisson iterates, the residual and the pressure agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# grid, lengths, y stretching: where the kernel's split can go wrong
BOXES = [((32, 16, 16), (8.0, 1.0, 1.0), None),     # whole V-cycle in it, 16 rows per block, halo of one block
         ((16, 8, 8), (2.0, 1.0, 1.0), 1.5),        # one block from the first level on
         ((7, 32, 32), (14.0, 2.0, 2.0), 1.5),      # odd row length, x never coarsened (natural storage)
         ((64, 64, 8), (4.0, 4.0, 0.5), 1.5),       # more rows per plane than per block (halo over many blocks)
         ((24, 20, 12), (2.4, 2.0, 1.2), None),     # coarsest level of 90 cells (inverse not staged)
         ((96, 12, 4), (16.0, 2.0, 0.5), 1.5),      # short rows of blocks, few planes
         ((64, 32, 32), (8.0, 1.0, 1.0), None),     # two cluster levels above the one-block ones
         ((128, 32, 32), (32.0, 1.0, 1.0), 1.5)]    # levels above it swept by separate launches


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,lengths,q", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_low_vcycle_is_bit_identical(shape, lengths, q, mode):
    from turbins_gb300 import api, build
    from turbins_gb300 import workload as W
    build.build()
    case = W.poisson_case(*shape, lengths, q)
    vel = W.fourier_velocity(case.grid, 7)
    out = []
    for tail in (None, 0):
        ctx = api.Context(case.grid, case.params)
        ctx.set_pressure_mode(api.PMODE_FP64 if mode == "fp64" else api.PMODE_MIXED)
        if tail is not None:
            ctx.set_mg_tail(tail)
        for f, k in ((api.F_U, "u"), (api.F_V, "v"), (api.F_W, "w")):
            ctx.upload(f, vel[k])
        ctx.upload(api.F_PHI, np.zeros(case.grid.shape))
        ctx.Pressure_set_RHS(1.0)
        it, rr = ctx.Pressure_solve()
        out.append((it, rr, ctx.download(api.F_PHI)))
        ctx.close()
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("shape,lengths,q", [((160, 96, 48), (16.0, 2.0, 2.0), 1.5),   # widths of z that differ in the last bits
                                             ((112, 80, 56), (4.0, 2.0, 1.0), None),   # rows and planes that leave blocks part empty
                                             ((128, 128, 64), (2.0, 2.0, 1.0), None)])  # planes alike
def test_fp64_column_sweeps_converge_as_fp32(shape, lengths, q):
    """The marching FP64 smoother and residual of the large levels: the same
    cycle as the FP32 one but for rounding, so as many CG iterations (one more
    or less) and the same pressure to the solves' tolerance."""
    from turbins_gb300 import api, build
    from turbins_gb300 import workload as W
    build.build()
    case = W.poisson_case(*shape, lengths, q)
    vel = W.fourier_velocity(case.grid, 11)
    out = []
    for mode in (api.PMODE_FP64, api.PMODE_MIXED):
        ctx = api.Context(case.grid, case.params)
        ctx.set_pressure_mode(mode)
        # the same sweeps in both modes
        ctx.set_mg_sweeps(4, 4)
        for f, k in ((api.F_U, "u"), (api.F_V, "v"), (api.F_W, "w")):
            ctx.upload(f, vel[k])
        ctx.upload(api.F_PHI, np.zeros(case.grid.shape))
        ctx.Pressure_set_RHS(1.0)
        it, rr = ctx.Pressure_solve()
        out.append((it, ctx.download(api.F_PHI)))
        ctx.close()
    assert abs(out[0][0] - out[1][0]) <= 1
    scale = np.abs(out[0][1]).max()
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-7 * scale
