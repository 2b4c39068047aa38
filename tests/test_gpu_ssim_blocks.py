"""Block SSIM windows and the smaller scales straight from the pictures, against the C restatement at the edges
of their tiles: 64 by 32 windows of 4 samples, 128 x 64 samples of the next scales, widths that leave part of
a vector, planes whose rows rule vector loads out, and values that are clipped as they are read."""
import numpy as np
import pytest

import oracle
import qmiv_b200

pytestmark = pytest.mark.gpu

MASK = oracle.SSIM | oracle.MSSSIM | oracle.IVMSSSIM
SUB = {420: (1, 1), 422: (1, 0), 444: (0, 0)}


def _pair(W, H, bd, cf, seed, over=False):
    rng = np.random.default_rng(seed)
    sx, sy = SUB[cf]
    top = (1 << bd) - 1
    dt = np.uint8 if bd <= 8 else np.uint16
    out = []
    for _ in range(2):
        planes = []
        for c in range(3):
            shape = (H >> sy, W >> sx) if c else (H, W)
            x = np.where(rng.random(shape) < 0.3, rng.choice([0, top], shape), rng.integers(0, top + 1, shape))
            if over:
                x = np.where(rng.random(shape) < 0.01, rng.integers(top + 1, np.iinfo(dt).max + 1, shape), x)
            planes.append(x.astype(dt))
        out.append(tuple(planes))
    return out


def _compare(got, exp):
    for k in ("ssim", "msssim", "ivmsssim"):
        assert (got[k][:3] if isinstance(got[k], list) else got[k]) == (exp[k][:3] if isinstance(exp[k], list) else exp[k]), k


# nx = W/4 - 1 and ny = H/4 - 1 windows at scale 0: 63, 64, 65 and 31, 32, 33 of them
@pytest.mark.parametrize("W,H", [(256, 128), (260, 132), (264, 136), (130, 178), (382, 254), (178, 258)])
@pytest.mark.parametrize("bd,cf", [(8, 420), (10, 420), (8, 422), (12, 422), (8, 444), (14, 444)])
def test_pair(W, H, bd, cf, qctx, oracle_lib):
    f0, f1 = _pair(W, H, bd, cf, W * 7 + H + bd)
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, cf), f0, f1, MASK)
    with qmiv_b200.Calc(qctx, W, H, bd, cf) as calc:
        _compare(calc.compute(f0, f1, MASK), exp)


@pytest.mark.parametrize("bd,cf", [(10, 420), (12, 444)])
def test_clipped(bd, cf, qctx, oracle_lib):
    W, H = 260, 180
    f0, f1 = _pair(W, H, bd, cf, 3, over=True)
    top = (1 << bd) - 1
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, cf), tuple(np.minimum(p, top) for p in f0),
                                  tuple(np.minimum(p, top) for p in f1), MASK)
    with qmiv_b200.Calc(qctx, W, H, bd, cf, invalid_pel_action=qmiv_b200.PEL_CNCL) as calc:
        _compare(calc.compute(f0, f1, MASK), exp)
