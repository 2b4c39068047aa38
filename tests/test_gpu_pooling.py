"""Pooling sums over rows and windows against the C restatement: lengths around the counts of threads that share
a chain, signed terms, and terms so far apart that the order of the additions matters."""
import numpy as np
import pytest

import oracle
import qmiv_b200

pytestmark = pytest.mark.gpu

# A window pair whose covariance all but cancels the constant of the contrast term: SSIM below 2^-32
TINY_R = [250, 4, 1, 7, 252, 249, 4, 254, 248, 248, 251, 249, 250, 6, 253, 253,
          1, 4, 3, 250, 254, 252, 252, 253, 4, 254, 0, 0, 0, 249, 4, 6,
          6, 0, 6, 5, 249, 7, 6, 251, 252, 250, 249, 5, 255, 3, 255, 4,
          2, 0, 252, 251, 254, 2, 0, 255, 4, 252, 248, 252, 2, 5, 5, 254]
TINY_T = {34: 36, 35: 21, 50: 28, 51: 16}


def _same(got, exp, keys):
    for k in keys:
        g, e = got[k], exp[k]
        assert (list(g[:3]) if isinstance(e, (list, tuple)) else g) == (list(e[:3]) if isinstance(e, (list, tuple)) else e), k


def _rows(W, H, bd, wide):
    """Row differences of one step in one sample at the pole, none, or (wide) full scale in every sample."""
    top = (1 << bd) - 1
    dt = np.uint8 if bd <= 8 else np.uint16
    rng = np.random.default_rng(W + H + bd)
    a = [np.zeros((H >> s, W >> s), dt) for s in (0, 1, 1)]
    b = [p.copy() for p in a]
    for p in b:
        h = p.shape[0]
        p[0, 3] = 1
        p[2:h - 1] = top if wide else rng.integers(0, 4, (h - 3, p.shape[1]))
    return tuple(a), tuple(b)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("W,H,bd", [(2048, 64, 14), (2048, 8, 8), (16, 254, 10), (16, 256, 10), (16, 258, 10), (16, 2050, 8), (16, 4100, 14)])
def test_rows(W, H, bd, wide, qctx, oracle_lib):
    f0, f1 = _rows(W, H, bd, wide)
    mask = oracle.PSNR | oracle.WSPSNR | oracle.IVPSNR | oracle.IVSSIM
    p = oracle.make_params(W, H, bd, 420, erp=True)
    exp = oracle_lib.compute_pair(p, f0, f1, mask)
    with qmiv_b200.Calc(qctx, W, H, bd, 420, erp=True) as calc:
        _same(calc.compute(f0, f1, mask), exp, ("wspsnr", "ivpsnr", "ivpsnr_r2t", "ivpsnr_t2r", "ivssim"))
        m = np.full((H, W), 255, np.uint8)
        m[:, ::3] = 1
        exp, n_exp = oracle_lib.compute_pair_masked(p, f0, f1, m, 8)
        got, n_got = calc.compute_masked(f0, f1, m, 8)
    assert n_got == n_exp
    _same(got, exp, ("wspsnr", "wspsnr_pic", "ivpsnr", "ivpsnr_r2t", "ivpsnr_t2r"))


@pytest.mark.parametrize("nx", [1, 2, 15, 16, 17, 127, 128, 129, 1023])
def test_windows(nx, qctx, oracle_lib):
    """Unrelated pictures: window values of both signs."""
    W, H = 4 * (nx + 1), 40
    rng = np.random.default_rng(nx)
    f0, f1 = [tuple(rng.integers(0, 256, (H >> s, W >> s)).astype(np.uint8) for s in (0, 1, 1)) for _ in range(2)]
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, 8, 420), f0, f1, oracle.SSIM)
    with qmiv_b200.Calc(qctx, W, H, 8, 420) as calc:
        _same(calc.compute(f0, f1, oracle.SSIM), exp, ("ssim",))


def test_tiny_window(qctx, oracle_lib):
    r = np.array(TINY_R, float)
    t = np.zeros(64)
    for k, v in TINY_T.items():
        t[k] = v
    cov = (r * t).mean() - r.mean() * t.mean()
    l = (2 * r.mean() * t.mean() + 6.5025) / (r.mean() ** 2 + t.mean() ** 2 + 6.5025)
    assert 0 < abs(l * (2 * cov + 58.5225) / (r.var() + t.var() + 58.5225)) < 2.0 ** -32
    W, H = 4096, 16
    f0, f1 = [tuple(np.full((H >> s, W >> s), 100, np.uint8) for s in (0, 1, 1)) for _ in range(2)]
    f0[0][4:12, 400:408] = r.reshape(8, 8)
    f1[0][4:12, 400:408] = t.reshape(8, 8)
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, 8, 420), f0, f1, oracle.SSIM)
    with qmiv_b200.Calc(qctx, W, H, 8, 420) as calc:
        _same(calc.compute(f0, f1, oracle.SSIM), exp, ("ssim",))


@pytest.mark.parametrize("H", [14, 16, 18, 254, 1030, 2050])
@pytest.mark.parametrize("at", [0.0, 0.4, 1.0])
def test_rows_whose_largest_comes_late(H, at, qctx, oracle_lib):
    """Rows of one step in one sample and, from the given share of the height on, two rows of full scale: chains
    that are summed in order, with prefixes of every length before the largest term."""
    W, bd = 2048, 14
    a = [np.zeros((H >> s, W >> s), np.uint16) for s in (0, 1, 1)]
    b = [p.copy() for p in a]
    for p in b:
        h = p.shape[0]
        p[:, 3] = 1
        y = int(at * (h - 2))
        p[y:y + 2] = (1 << bd) - 1
    f0, f1 = tuple(a), tuple(b)
    mask = oracle.WSPSNR | oracle.IVPSNR
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, 420, erp=True), f0, f1, mask)
    with qmiv_b200.Calc(qctx, W, H, bd, 420, erp=True) as calc:
        _same(calc.compute(f0, f1, mask), exp, ("wspsnr", "ivpsnr", "ivpsnr_r2t", "ivpsnr_t2r"))
