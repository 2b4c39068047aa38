"""Gaussian SSIM windows against the C restatement where their arithmetic and launch shapes change: the largest
samples whose products are exact, deeper ones, the 65535 margin, samples above the maximum, and sizes around
the tiles of either window count per lane."""
import numpy as np
import pytest

import oracle
import qmiv_b200

pytestmark = pytest.mark.gpu


def _frames(W, H, bd, seed, top):
    """Samples at and near both ends of the range, full scale in every window."""
    rng = np.random.default_rng(seed)
    dt = np.uint8 if bd <= 8 else np.uint16
    return [tuple(np.where(rng.random((H >> s, W >> s)) < 0.5, rng.integers(0, top + 1, (H >> s, W >> s)),
                           rng.choice([0, 1, top - 1, top], (H >> s, W >> s))).astype(dt) for s in (0, 1, 1)) for _ in range(2)]


@pytest.mark.parametrize("W,H", [(22, 22), (202, 42), (204, 40), (266, 44), (394, 60)])
@pytest.mark.parametrize("bd", [8, 10, 14, 15, 16])
@pytest.mark.parametrize("mode,border,stride", [(0, 0, 1), (0, 4, 1), (0, 1, 3), (0, 3, 4), (1, 0, 1)])
def test_window_values(W, H, bd, mode, border, stride, qctx, oracle_lib):
    f0, f1 = _frames(W, H, bd, 1000 * bd + W, (1 << bd) - 1)
    exp = oracle_lib.compute_pair_ssim(oracle.make_params(W, H, bd, 420), f0, f1, mode, border, 11, stride, oracle.SSIM)
    with qmiv_b200.Calc(qctx, W, H, bd, 420, ssim_mode=mode, ssim_border=border, ssim_stride=stride) as calc:
        got = calc.compute(f0, f1, oracle.SSIM)
    assert got["ssim"] == exp["ssim"]


@pytest.mark.parametrize("action", [qmiv_b200.PEL_SKIP, qmiv_b200.PEL_CNCL])
def test_samples_above_the_maximum(action, qctx, oracle_lib):
    W, H, bd = 130, 48, 10
    f0, f1 = _frames(W, H, bd, 5, 1023)
    f0[0][11, 17] = 65535
    f1[2][3, 9] = 40001
    ref = [f0, f1] if action == qmiv_b200.PEL_SKIP else [tuple(np.minimum(p, 1023) for p in f) for f in (f0, f1)]
    exp = oracle_lib.compute_pair_ssim(oracle.make_params(W, H, bd, 420), *ref, 0, 0, 11, 1, oracle.SSIM)
    with qmiv_b200.Calc(qctx, W, H, bd, 420, ssim_mode=0, ssim_stride=1, invalid_pel_action=action) as calc:
        got = calc.compute(f0, f1, oracle.SSIM)
    assert got["ssim"] == exp["ssim"]
