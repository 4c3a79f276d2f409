"""Which grids the weight gradient takes, and its numbers on all that it does:
padded lines that do not fill the 128 positions of a tile, also in the form
with one x tap per CTA, and the refusal of grids whose voxel tile is no
multiple of 16."""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(U.to_blocked(a), dtype=np.float32)).to(torch.bfloat16).cuda()


def _run(X, Y, Z, cin, cout):
    from turbins_gb300 import build
    build.build()
    from turbins_gb300 import net as N
    rng = np.random.default_rng(X + 7 * Y + cin)
    x, dy = (U.bf16_round(rng.normal(size=(c, Z, Y, X))) for c in (cin, cout))
    dw = torch.zeros((27, cout, cin), dtype=torch.float32, device="cuda")
    N.conv3_wgrad(X, Y, Z, cin, cout, _dev(x), _dev(dy), dw)
    return x, dy, dw.cpu().numpy()


@pytest.mark.parametrize("X,Y,Z,cin,cout", [(112, 5, 6, 16, 16), (48, 9, 7, 32, 16), (144, 3, 5, 16, 32), (80, 4, 30, 32, 32),
                                            (112, 64, 120, 16, 16), (48, 6, 5, 64, 32), (16, 16, 8, 128, 64)])
def test_wgrad_numbers(X, Y, Z, cin, cout):
    x, dy, dw = _run(X, Y, Z, cin, cout)
    # FP32 sums of exact BF16 products: bounded by the sum of |terms|
    bound = 1e-5 * U.conv3_wgrad(np.abs(x), np.abs(dy)) + 1e-6
    assert np.all(np.abs(dw - U.conv3_wgrad(x, dy)) <= bound)


@pytest.mark.parametrize("X,Y,Z,cin,cout", [(62, 8, 21, 16, 32), (126, 2, 3, 32, 32), (24, 24, 8, 64, 64), (3, 2, 2, 16, 16)])
def test_wgrad_refuses_ragged_tiles(X, Y, Z, cin, cout):
    with pytest.raises(RuntimeError, match="no multiple of 16"):
        _run(X, Y, Z, cin, cout)
