"""Row sums, totals and the GCD against the C restatement where the prepass changes its loads and its arithmetic:
rows that start anywhere in 16 bytes, few and many vectors per lane, samples from 2^14 up, clipped and invalid ones."""
import numpy as np
import pytest

import oracle
import qmiv_b200

pytestmark = pytest.mark.gpu

MASK = oracle.PSNR | oracle.WSPSNR | oracle.IVPSNR
KEYS = ("psnr", "wspsnr", "ivpsnr", "gcd_r2t")


def _pair(W, H, bd, cf, top):
    rng = np.random.default_rng(W * 31 + bd)
    dt = np.uint8 if bd <= 8 else np.uint16
    sh = [(H, W)] + 2 * [(H >> (cf == 420), W >> (cf != 444))]
    return [tuple(np.where(rng.random(s) < 0.3, rng.choice([0, top], s), rng.integers(0, top + 1, s)).astype(dt) for s in sh) for _ in range(2)]


def _check(got, exp):
    for k in KEYS:
        assert (list(got[k][:3]) if isinstance(exp[k], (list, tuple)) else got[k]) == (list(exp[k][:3]) if isinstance(exp[k], (list, tuple)) else exp[k]), k


@pytest.mark.parametrize("W", [8, 22, 130, 254, 1028, 2062])
@pytest.mark.parametrize("bd,cf", [(8, 420), (8, 444), (10, 420), (14, 422), (15, 420), (16, 444)])
def test_rows(W, bd, cf, qctx, oracle_lib):
    H = 18
    f0, f1 = _pair(W, H, bd, cf, (1 << bd) - 1)
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, cf, erp=True), f0, f1, MASK)
    with qmiv_b200.Calc(qctx, W, H, bd, cf, erp=True) as calc:
        _check(calc.compute(f0, f1, MASK), exp)


@pytest.mark.parametrize("W,bd,top", [(134, 10, 1024), (134, 10, 65535), (256, 12, 20000), (70, 6, 255)])
@pytest.mark.parametrize("action", [qmiv_b200.PEL_SKIP, qmiv_b200.PEL_CNCL, qmiv_b200.PEL_STOP])
def test_invalid(W, bd, top, action, qctx, oracle_lib):
    H = 12
    f0, f1 = _pair(W, H, bd, 420, (1 << bd) - 1)
    f1[1][2, W // 2 - 3] = top
    f0[0][5, 7] = top
    with qmiv_b200.Calc(qctx, W, H, bd, 420, erp=True, invalid_pel_action=action) as calc:
        if action == qmiv_b200.PEL_STOP:
            with pytest.raises(qmiv_b200.QmivError):
                calc.compute(f0, f1, MASK)
            return
        got = calc.compute(f0, f1, oracle.PSNR | oracle.WSPSNR)
    m = (1 << bd) - 1
    ref = [f0, f1] if action == qmiv_b200.PEL_SKIP else [tuple(np.minimum(p, m) for p in f) for f in (f0, f1)]
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, 420, erp=True), *ref, oracle.PSNR | oracle.WSPSNR)
    for k in ("psnr", "wspsnr"):
        assert list(got[k][:3]) == list(exp[k][:3]), k
