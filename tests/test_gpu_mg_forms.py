"""Every form of the V-cycle's kernels against the plain one (a launch per half
sweep, a thread per cell): the same operations per cell in the same order, so
the Poisson iterates, the residual and the pressure are the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64, MIXED = 0, 1


@pytest.fixture(scope="module")
def api():
    from turbins_gb300 import api as A
    from turbins_gb300 import build
    build.build()
    return A


def solve(api, case, vel, mode, forms=None, tail=None):
    """(iterations, residual, pressure), launches of the solve"""
    ctx = api.Context(case.grid, case.params)
    ctx.set_pressure_mode(mode)
    if forms is not None:
        ctx.set_mg_forms(*forms)
    if tail is not None:
        ctx.set_mg_tail(tail)
    for f, k in ((api.F_U, "u"), (api.F_V, "v"), (api.F_W, "w")):
        ctx.upload(f, vel[k])
    ctx.upload(api.F_PHI, np.zeros(case.grid.shape))
    ctx.Pressure_set_RHS(1.0)
    n0 = api.kernel_launches(ctx)
    it, rr = ctx.Pressure_solve()
    n = api.kernel_launches(ctx) - n0
    phi = ctx.download(api.F_PHI)
    ctx.close()
    return (it, rr, phi), n


def same(a, b):
    return a[:2] == b[:2] and np.array_equal(a[2], b[2])


def problem(shape, lengths, q, zw=None):
    from turbins_gb300 import workload as W
    case = W.poisson_case(*shape, lengths, q)
    if zw is not None:
        case.grid.zw = np.concatenate([[0.0], np.cumsum(zw), [np.sum(zw) + zw[-1]]])[:shape[2] + 1]
        case.grid.zc = np.append(0.5 * (case.grid.zw[1:] + case.grid.zw[:-1]), case.grid.zw[-1] + 0.5 * zw[-1])
    return case, W.fourier_velocity(case.grid, 5)


# the single-block launch over global memory (k_vcycle_tail): from the first
# level on; below a level of its own; odd extents, x never coarsened; a level
# that the shared-memory kernel refuses (2400 cell pairs for one block)
TAIL = [((24, 12, 8), (3.0, 1.0, 1.0), 1.5), ((32, 32, 16), (4.0, 2.0, 2.0), None), ((7, 20, 16), (14.0, 2.0, 2.0), 1.5),
        ((5, 40, 20), (10.0, 2.0, 1.0), None)]


@pytest.mark.parametrize("mode", [FP64, MIXED])
@pytest.mark.parametrize("shape,lengths,q", TAIL, ids=["x".join(map(str, t[0])) for t in TAIL])
def test_single_block_tail(api, shape, lengths, q, mode):
    case, vel = problem(shape, lengths, q)
    plain, n0 = solve(api, case, vel, mode, tail=0)
    tail, n = solve(api, case, vel, mode, forms=(0, True))
    assert same(plain, tail)
    assert n < n0   # it ran: a launch in place of many
    assert same(plain, solve(api, case, vel, mode)[0])


# the shared-memory cluster where the device holds only 8 blocks, or no cluster
LOW = [((32, 16, 16), (8.0, 1.0, 1.0), None), ((7, 32, 32), (14.0, 2.0, 2.0), 1.5), ((64, 64, 8), (4.0, 4.0, 0.5), 1.5),
       ((64, 32, 16), (8.0, 1.0, 1.0), 1.5)]


@pytest.mark.parametrize("mode", [FP64, MIXED])
@pytest.mark.parametrize("blocks", [1, 8])
@pytest.mark.parametrize("shape,lengths,q", LOW, ids=["x".join(map(str, t[0])) for t in LOW])
def test_fewer_cluster_blocks(api, shape, lengths, q, blocks, mode):
    case, vel = problem(shape, lengths, q)
    plain, n0 = solve(api, case, vel, mode, tail=0)
    low, n = solve(api, case, vel, mode, forms=(blocks, True))
    assert same(plain, low)
    assert n < n0


# the FP64 kernels that march columns (304 blocks or more): 8 planes per block
# and 3 left over, 2 planes and 1, odd nx (only the residual marches), and z
# widths that repeat, change within a block and repeat again (the kept
# coefficients are formed anew where a plane's differ)
def steps(nz, runs):
    """nz widths: runs of (count, width), over and over"""
    out = []
    while len(out) < nz:
        for n, w in runs:
            out += [w] * n
    return np.array(out[:nz])


COLUMNS = [((256, 128, 43), (4.0, 2.0, 21.5), None, None),
           ((128, 96, 27), (4.0, 2.0, 13.5), 1.5, None),
           ((63, 128, 64), (31.5, 2.0, 1.0), None, None),
           ((256, 128, 48), (4.0, 2.0, 1.0), None, steps(48, [(3, 0.02), (1, 0.03), (5, 0.02), (2, 0.025), (2, 0.02)])),
           ((256, 96, 48), (4.0, 2.0, 1.0), 1.5, steps(48, [(1, 0.02), (1, 0.03)])),
           ((192, 96, 64), (4.0, 2.0, 1.0), None, 0.02 * 1.01 ** np.arange(64))]


@pytest.mark.parametrize("shape,lengths,q,zw", COLUMNS, ids=["x".join(map(str, t[0])) for t in COLUMNS])
def test_fp64_columns(api, shape, lengths, q, zw):
    case, vel = problem(shape, lengths, q, zw)
    assert same(solve(api, case, vel, FP64, forms=(16, False))[0], solve(api, case, vel, FP64)[0])


def test_forms_are_checked(api):
    from turbins_gb300 import workload as W
    case = W.poisson_case(16, 8, 8, (2.0, 1.0, 1.0))
    ctx = api.Context(case.grid, case.params)
    for bad in (-1, 2, 4, 32):
        with pytest.raises(api.TurbError):
            ctx.set_mg_forms(bad)
    ctx.close()
