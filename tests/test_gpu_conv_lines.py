"""The 3x3x3 convolutions where their tiles can go wrong: x extents that do
not fill a 128-position tile of the padded line, rings longer than the
accumulator ring, single-row items, channel counts that leave a partial chunk,
output channels split over CTAs."""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 1, 1, 16, 16), (8, 2, 2, 16, 32), (62, 3, 21, 32, 16), (64, 9, 40, 16, 16), (126, 2, 3, 32, 32),
          (130, 3, 2, 16, 16), (160, 5, 3, 32, 32), (128, 41, 2, 16, 32), (256, 3, 19, 16, 16),
          (4, 2, 2, 128, 128), (20, 6, 5, 96, 48), (40, 12, 10, 32, 64), (66, 8, 5, 48, 16), (130, 2, 3, 64, 64),
          (64, 24, 24, 64, 64)]


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(U.to_blocked(a), dtype=np.float32)).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("X,Y,Z,cin,cout", SHAPES)
def test_conv_tiles(X, Y, Z, cin, cout):
    from turbins_gb300 import build
    build.build()
    from turbins_gb300 import net as N
    rng = np.random.default_rng(X * 31 + Y * 7 + cin)
    W = rng.normal(0, 0.2, size=(27, cout, cin)).astype(np.float32)
    b = rng.normal(0, 0.1, size=cout).astype(np.float32)
    Wd, Wq = torch.from_numpy(W).cuda(), U.bf16_round(W)
    for dgrad, ci, co in ((False, cin, cout), (True, cout, cin)):
        x = U.bf16_round(rng.normal(size=(ci, Z, Y, X)))
        # guard elements either side: nothing outside the output is written
        n = co * X * Y * Z
        buf = torch.full((n + 128,), 7.0, dtype=torch.bfloat16, device="cuda")
        out = buf[64:64 + n].view(co // 8, Z, Y, X, 8)
        N.conv3(X, Y, Z, cin, cout, _dev(x), Wd, None if dgrad else torch.from_numpy(b).cuda(), relu=not dgrad,
                dgrad=dgrad, out=out)
        got = U.from_blocked(out.float().cpu().numpy().astype(np.float64), co)
        ref = U.conv3_dgrad(x, Wq) if dgrad else np.maximum(U.conv3(x, Wq, b.astype(np.float64)), 0.0)
        # one BF16 rounding; FP32 sums of at most 3456 exact products
        assert np.all(np.abs(got - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-5 * np.abs(ref).max())
        assert bool((buf[:64] == 7).all()) and bool((buf[64 + n:] == 7).all())


@pytest.mark.parametrize("shift", range(8))
def test_umma_swizzle128_mn_row_shift(shift):
    from turbins_gb300 import build
    build.build()
    from turbins_gb300 import net as N
    assert N.selftest_umma(3, shift) == 0


@pytest.mark.parametrize("X,Y,Z,cin,cout", [(16, 1, 1, 16, 16), (8, 2, 3, 32, 32), (64, 7, 9, 16, 16), (62, 8, 21, 16, 32),
                                            (128, 5, 3, 16, 16), (256, 3, 2, 32, 32), (160, 4, 5, 32, 16),
                                            (128, 64, 100, 16, 16)])
def test_wgrad_tiles(X, Y, Z, cin, cout):
    from turbins_gb300 import build
    build.build()
    from turbins_gb300 import net as N
    rng = np.random.default_rng(X + 5 * Y + cout)
    x, dy = (U.bf16_round(rng.normal(size=(c, Z, Y, X))) for c in (cin, cout))
    dw = torch.zeros((27, cout, cin), dtype=torch.float32, device="cuda")
    try:
        N.conv3_wgrad(X, Y, Z, cin, cout, _dev(x), _dev(dy), dw)
    except RuntimeError:
        # voxel tiles that are no multiple of 16 are refused
        bx = min(X, 128)
        by = min(Y, 128 // bx)
        assert bx * by * min(Z, 128 // (bx * by)) % 16
        return
    # FP32 sums of exact BF16 products: bounded by the sum of |terms|
    bound = 1e-5 * U.conv3_wgrad(np.abs(x), np.abs(dy)) + 1e-6
    assert np.all(np.abs(dw.cpu().numpy() - U.conv3_wgrad(x, dy)) <= bound)
