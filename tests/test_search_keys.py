"""The 4:2:0 search's integer keys at the limits of bit depth, weights, GCD bound and mask values: the host's
conditions against exact integers (CPU), and results on both sides of each limit against the C restatement."""
import ctypes

import numpy as np
import pytest

import oracle
import qmiv_b200
from qmiv_b200 import _lib

WEIGHTS = [(4, 1, 1), (2, 1, 1), (1, 1, 1), (1, 0, 0), (0, 1, 1), (0, 0, 1), (0, 0, 0), (20, 1, 3), (500, 100, 100)]


def _keys(R, maxv, w, g):
    a3 = ctypes.c_int32 * 3
    out = _lib.QmivCpsKeys()
    _lib.check(qmiv_b200.library().qmiv_probe_cps_keys(R, maxv, a3(*w), a3(*g), ctypes.byref(out)), "qmiv_probe_cps_keys")
    return out


def _bounds(maxv):
    return [(g, g, g) for g in sorted({0, 1, maxv // 100, maxv // 10, maxv // 4, maxv // 3, maxv // 2, maxv})] + [(maxv // 100, 0, maxv // 4)]


@pytest.mark.parametrize("bd", range(8, 17))
def test_admitted_keys_hold_every_error(bd):
    """Where the keys are admitted: no key leaves 32 bits or borrows from the code, a masked sample's key is above
    every real one, and a warp's masked row sums stay within the 32 bits they are formed in."""
    maxv = (1 << bd) - 1
    admitted = 0
    for R in range(1, 6):
        D, code = 2 * R + 1, (3 + 2 * R) * (2 * R + 1) + 3 + 2 * R
        for w in WEIGHTS:
            for g in _bounds(maxv):
                k = _keys(R, maxv, w, g)
                K, m = 1 << k.key_bits, k.mid
                assert K >= D * D and (not k.masked or k.shared)
                if not k.shared:
                    continue
                ext = lambda c: [(s, r) for s in (-g[c] - m, maxv + g[c] - m) for r in (-m, maxv - m)]   # test, candidate less mid
                part = [[w[c] * (r * r - 2 * s * r) for s, r in ext(c)] for c in range(3)]              # extremes of a convex-concave form
                inner = [[w[c] * (r * r - 2 * s * r) for s in (-g[c] - m, maxv + g[c] - m) for r in (max(-m, min(maxv - m, s)),)] for c in range(3)]
                low, high = sum(min(p + q) for p, q in zip(part, inner)), sum(max(p) for p in part)
                assert K * (low + k.bias) >= 0 and K * (high + k.bias) + code < 1 << 32
                if not k.masked:
                    continue
                admitted += 1
                chroma_low, chroma_high = sum(min(part[c] + inner[c]) for c in (1, 2)), sum(max(part[c]) for c in (1, 2))
                assert k.masked_value + K * (k.bias + chroma_low) > K * (high + k.bias) + code
                assert k.masked_value + K * (k.bias + chroma_high) + code < 1 << 32
                # four pixels of a lane, 32 lanes; mask samples of 16 bits
                term = 4 * max(maxv + x for x in g) ** 2 * 65535
                assert 32 * (term >> k.sum_split) < 1 << 32 and 32 * ((1 << k.sum_split) - 1) < 1 << 32
    assert admitted or bd > 13


# bit depth, weights, share of the maximum that bounds the GCD, search range: both sides of a limit
LIMITS = [(12, (2, 1, 1, 0), 0.01, 2), (12, (2, 1, 1, 0), 0.15, 2), (12, (2, 1, 1, 0), 0.16, 2), (12, (1, 1, 1, 0), 0.01, 1),
          (12, (1, 1, 1, 0), 0.26, 2), (12, (1, 1, 1, 0), 0.27, 2), (13, (1, 0, 0, 0), 0.0, 2), (13, (1, 0, 0, 0), 0.01, 2),
          (13, (0, 0, 0, 0), 0.0, 5), (11, (4, 1, 1, 0), 0.41, 3), (11, (4, 1, 1, 0), 0.42, 3), (12, (4, 1, 1, 0), 0.15, 2),
          (12, (4, 1, 1, 0), 0.16, 2), (11, (4, 1, 1, 0), 0.15, 4), (11, (4, 1, 1, 0), 0.16, 4), (8, (500, 100, 100, 0), 0.01, 2)]


def _regions(bd, W=520, H=36):
    """Frames whose samples are all 0 or the maximum: In0 and In1 opposite in sign in two regions wider than a tile, a strip at random."""
    top, dt = (1 << bd) - 1, np.uint8 if bd == 8 else np.uint16
    rng = np.random.default_rng(bd)
    f0, f1 = [], []
    for s in (0, 1, 1):
        h, w = H >> s, W >> s
        a, b = np.zeros((h, w), np.int64), np.full((h, w), top)
        a[:, :w // 3], b[:, :w // 3] = top, 0
        a[h - 4:, :], b[h - 4:, :] = rng.choice([0, top], (4, w)), rng.choice([0, top], (4, w))
        f0.append(a.astype(dt)); f1.append(b.astype(dt))
    return tuple(f0), tuple(f1)


@pytest.mark.gpu
@pytest.mark.parametrize("bd,cws,unc,R", LIMITS)
def test_masked_search_at_the_limits(bd, cws, unc, R, qctx, oracle_lib):
    """Full-scale masks of 8 to 14 bits, and a mask whose samples exceed its bit depth."""
    f0, f1 = _regions(bd)
    H, W = f0[0].shape
    for mbd, top in ((14, 16383), (8, 255), (10, 65535)):
        m = np.full((H, W), top, np.uint8 if mbd == 8 else np.uint16)
        m[:, W - 40:W - 8] = 0
        exp, nnm = oracle_lib.compute_pair_masked(oracle.make_params(W, H, bd, 420, search_range=R, cws=cws, unc=(unc, unc, unc, 0.0)),
                                                  f0, f1, m, mbd)
        with qmiv_b200.Calc(qctx, W, H, bd, 420, search_range=R, cws=cws, unc=(unc, unc, unc, 0.0)) as calc:
            got, n = calc.compute_masked(f0, f1, m, mbd, qmiv_b200.IVPSNR)
        assert n == nnm
        for k in ("gcd_r2t", "ivpsnr", "ivpsnr_r2t", "ivpsnr_t2r"):
            assert got[k] == exp[k], (mbd, k)


@pytest.mark.gpu
@pytest.mark.parametrize("bd,cws,unc,R", LIMITS)
def test_search_at_the_limits(bd, cws, unc, R, qctx, oracle_lib):
    f0, f1 = _regions(bd)
    H, W = f0[0].shape
    kw = dict(search_range=R, cws=cws, unc=(unc, unc, unc, 0.0))
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, 420, **kw), f0, f1, oracle.IVPSNR | oracle.IVSSIM)
    with qmiv_b200.Calc(qctx, W, H, bd, 420, **kw) as calc:
        got = calc.compute(f0, f1, oracle.IVPSNR | oracle.IVSSIM)
    assert {k: got[k] for k in exp} == exp
