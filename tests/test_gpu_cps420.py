"""The 4:2:0 corresponding-pixel-shift search against the C restatement where its tiles, keys and paths
change: pictures smaller than a tile, one sample past a tile edge, every search range, the largest bit
depth of the integer keys and the depths past it, invalid samples, planes TMA cannot take."""
import numpy as np
import pytest

import oracle
import qmiv_b200
from qmiv_b200 import synth

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (10, 8), (126, 14), (128, 16), (130, 18), (262, 34)]


def _check(qctx, oracle_lib, shape, f0, f1, dev, metrics=None, **kw):
    W, H, bd, R = shape
    metrics = metrics or oracle.IVPSNR | (oracle.IVSSIM if min(W, H) >= 8 else 0) | (oracle.IVMSSSIM if min(W, H) >= 32 else 0)
    exp = oracle_lib.compute_pair(oracle.make_params(W, H, bd, 420, search_range=R), f0, f1, metrics)
    with qmiv_b200.Calc(qctx, W, H, bd, 420, search_range=R, **kw) as calc:
        got = calc.compute(dev(f0), dev(f1), metrics)
    assert {k: got[k] for k in exp} == exp


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("bd,R", [(8, 1), (8, 2), (10, 2), (10, 3), (8, 4), (10, 5), (11, 4), (12, 2), (12, 3), (14, 2)])
def test_tiles_keys_and_ranges(size, bd, R, qctx, oracle_lib):
    f0, f1 = synth.make_pair(*size, bd, seed=7 * bd + R, shift_range=R, texture_sigma=40.0, offset=(3, -2, 2))
    _check(qctx, oracle_lib, (*size, bd, R), f0, f1, lambda f: f)


@pytest.mark.parametrize("size", SIZES[1:])
@pytest.mark.parametrize("bd,top", [(8, 255), (10, 1023), (12, 4095)])
def test_extreme_samples(size, bd, top, qctx, oracle_lib):
    """Only the smallest and largest sample values: the widest keys, equal errors everywhere, clipped SCP samples."""
    rng = np.random.default_rng(bd)
    dt = np.uint8 if bd == 8 else np.uint16
    f = [tuple((rng.integers(0, 2, (size[1] >> s, size[0] >> s)) * top).astype(dt) for s in (0, 1, 1)) for _ in range(2)]
    _check(qctx, oracle_lib, (*size, bd, 2), f[0], f[1], lambda x: x)


@pytest.mark.parametrize("size,R", [((130, 18), 2), ((262, 34), 3)])
def test_samples_above_the_maximum(size, R, qctx, oracle_lib):
    """SKIP searches them as they are (literal int32 arithmetic); CNCL clips them first."""
    f0, f1 = synth.make_pair(*size, 10, seed=3)
    hot = [tuple(p.copy() for p in f) for f in (f0, f1)]
    hot[0][0][5, 7] = 40000
    hot[1][1][3, 2] = 65535
    _check(qctx, oracle_lib, (*size, 10, R), hot[0], hot[1], lambda f: f, metrics=oracle.IVPSNR,
           invalid_pel_action=qmiv_b200.PEL_SKIP)   # window moments of samples above 14 bits wrap and are not compared
    clipped = [tuple(np.minimum(p, 1023) for p in f) for f in hot]
    exp = oracle_lib.compute_pair(oracle.make_params(*size, 10, 420, search_range=R), *clipped, oracle.IVPSNR | oracle.IVSSIM)
    with qmiv_b200.Calc(qctx, *size, 10, 420, search_range=R, invalid_pel_action=qmiv_b200.PEL_CNCL) as calc:
        got = calc.compute(*hot, oracle.IVPSNR | oracle.IVSSIM)
    assert all(got[k] == exp[k] for k in exp if k != "invalid_pel")


@pytest.mark.parametrize("bd", [8, 10])
def test_planes_without_tma(bd, qctx, oracle_lib):
    """Device planes whose pitch is no multiple of 16 bytes are loaded sample by sample."""
    import torch
    def dev(frame):
        out = []
        for p in frame:
            t = torch.zeros(p.shape[0], p.shape[1] + 3, dtype=torch.uint8 if bd == 8 else torch.uint16, device="cuda")
            t[:, :p.shape[1]] = torch.from_numpy(np.ascontiguousarray(p)).cuda()
            out.append(t[:, :p.shape[1]])
        return tuple(out)
    f0, f1 = synth.make_pair(262, 50, bd, seed=11)
    _check(qctx, oracle_lib, (262, 50, bd, 2), f0, f1, dev)


@pytest.mark.parametrize("size", SIZES[1:])
@pytest.mark.parametrize("bd,mbd,R", [(8, 8, 2), (10, 8, 2), (10, 10, 1), (10, 14, 5), (11, 8, 3), (11, 12, 4), (12, 8, 2)])
def test_masked_tiles(size, bd, mbd, R, qctx, oracle_lib):
    """The masked search: single kept samples, weights over the mask's range, extreme picture samples, the
    depths at which a masked sample's key still fits and those past it; aligned and unaligned device planes."""
    import torch
    W, H = size
    rng = np.random.default_rng(bd * 100 + mbd + R)
    top, dt, mdt = (1 << bd) - 1, np.uint8 if bd == 8 else np.uint16, np.uint8 if mbd == 8 else np.uint16
    f = [tuple(np.where(rng.random((H >> s, W >> s)) < 0.5, rng.integers(0, top + 1, (H >> s, W >> s)),
                        rng.choice([0, top], (H >> s, W >> s))).astype(dt) for s in (0, 1, 1)) for _ in range(2)]
    m = np.where(rng.random((H, W)) < 0.3, rng.integers(1, 1 << mbd, (H, W)), 0).astype(mdt)
    m[0, 0] = m[H - 1, W - 1] = (1 << mbd) - 1
    exp, nnm = oracle_lib.compute_pair_masked(oracle.make_params(W, H, bd, 420, search_range=R, erp=True), *f, m, mbd)
    def dev(a, extra):
        t = torch.zeros(a.shape[0], a.shape[1] + extra, dtype=torch.uint8 if a.dtype == np.uint8 else torch.uint16, device="cuda")
        t[:, :a.shape[1]] = torch.from_numpy(np.ascontiguousarray(a)).cuda()
        return t[:, :a.shape[1]]
    with qmiv_b200.Calc(qctx, W, H, bd, 420, search_range=R, erp=True) as calc:
        for planes in ((*f, m), (*[tuple(dev(p, 5) for p in x) for x in f], dev(m, 3)), (*[tuple(dev(p, -p.shape[1] % 16) for p in x) for x in f], dev(m, -W % 16))):
            got, n = calc.compute_masked(*planes, mbd)
            assert n == nnm and {k: got[k] for k in exp} == exp


@pytest.mark.parametrize("size", [(262, 34), (520, 66), (392, 50)])
@pytest.mark.parametrize("bd,mbd,R", [(8, 8, 1), (10, 8, 2), (10, 10, 2), (8, 8, 3), (10, 12, 4), (10, 8, 5)])
def test_masked_tiles_and_strips_without_pixels(size, bd, mbd, R, qctx, oracle_lib):
    """Tiles of 128 x 16 and strips of 128 x 4 pixels whose mask is zero are skipped, one kept pixel at any of their
    corners keeps them: the first, last and inner tiles empty, single pixels, strips past the picture; planes with and
    without TMA, one pair and batches that mix them."""
    import torch
    W, H = size
    rng = np.random.default_rng(bd * 10 + R + W)
    top, dt, mdt = (1 << bd) - 1, np.uint8 if bd == 8 else np.uint16, np.uint8 if mbd == 8 else np.uint16
    f = [tuple(rng.integers(0, top + 1, (H >> s, W >> s)).astype(dt) for s in (0, 1, 1)) for _ in range(2)]
    def at(*pixels):
        m = np.zeros((H, W), mdt)
        for y, x in pixels:
            m[y, x] = rng.integers(1, 1 << mbd)
        return m
    block = np.zeros((H, W), mdt)
    block[17:30, 130:250] = 3
    last = np.zeros((H, W), mdt)
    last[(H - 1) // 16 * 16:, (W - 1) // 128 * 128:] = (1 << mbd) - 1
    masks = [at((0, 0)), at((H - 1, W - 1)), at((15, 127), (16, 128)), at((3, 128), (4, 127), (H - 1, 0)), block, last]
    def dev(a, extra):
        t = torch.zeros(a.shape[0], a.shape[1] + extra, dtype=torch.uint8 if a.dtype == np.uint8 else torch.uint16, device="cuda")
        t[:, :a.shape[1]] = torch.from_numpy(np.ascontiguousarray(a)).cuda()
        return t[:, :a.shape[1]]
    odd = [tuple(dev(p, 5) for p in x) for x in f]
    even = [tuple(dev(p, -p.shape[1] % 16) for p in x) for x in f]
    exp = [oracle_lib.compute_pair_masked(oracle.make_params(W, H, bd, 420, search_range=R), *f, m, mbd) for m in masks]
    want = lambda got, e: {k: got[k] for k in e} == e
    with qmiv_b200.Calc(qctx, W, H, bd, 420, search_range=R) as calc:
        for m, (e, n) in zip(masks, exp):
            for planes, extra in ((odd, 3), (even, -W % 16)):
                got, nnm = calc.compute_masked(*planes, dev(m, extra), mbd)
                assert nnm == n and want(got, e)
    pairs = [dict(frame0=p[0], frame1=p[1], width=W, height=H, bitdepth=bd, search_range=R, metrics="PSNR,WSPSNR,IVPSNR")
             for _ in masks for p in (odd, even)]
    with qmiv_b200.Batch(qctx, len(pairs), len(pairs) * W * H) as b:
        got, nnm = b.compute_masked(pairs, [dev(m, x) for m in masks for x in (3, -W % 16)], [mbd] * len(pairs))
    assert all(nnm[i] == exp[i // 2][1] and want(got[i], exp[i // 2][0]) for i in range(len(pairs)))


@pytest.mark.parametrize("R", [1, 2, 3, 5])
def test_work_list_with_and_without_tma(R, qctx, oracle_lib):
    """One launch over pairs that TMA can and cannot load, in turn: the copies of a tile are issued while the tile
    before it is searched, whichever way that one was loaded."""
    import torch
    W, H, bd = 390, 50, 10
    f = [synth.make_pair(W, H, bd, seed=20 + i, shift_range=R) for i in range(5)]
    exp = [oracle_lib.compute_pair(oracle.make_params(W, H, bd, 420, search_range=R), *p, oracle.IVPSNR | oracle.IVSSIM) for p in f]
    def dev(a, extra):
        t = torch.zeros(a.shape[0], a.shape[1] + extra, dtype=torch.uint16, device="cuda")
        t[:, :a.shape[1]] = torch.from_numpy(np.ascontiguousarray(a)).cuda()
        return t[:, :a.shape[1]]
    pairs = []
    for i, p in enumerate(f):
        a, b = [tuple(dev(x, 3 if i % 2 else -x.shape[1] % 16) for x in fr) for fr in p]
        pairs.append(dict(frame0=a, frame1=b, width=W, height=H, bitdepth=bd, search_range=R, metrics=["IVPSNR", "IVSSIM"]))
    with qmiv_b200.Batch(qctx, 40, 40 * W * H) as b:
        got = b.compute(pairs * 8)
    assert all({k: got[i][k] for k in exp[i % 5]} == exp[i % 5] for i in range(40))
