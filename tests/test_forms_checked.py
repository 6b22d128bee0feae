"""The affine DP's forms one after the other, for the gap scores that reach them: the
tagged 16-bit form with its handoff to the checked form and to 32-bit lanes (gaps of
-11 / -2 by name), and the untagged forms (a first gap of -32 does not fit the tags).
Both walks of the traceback (a warp a pair in batches up to 131072, a thread beyond)
meet regions of both lane widths.  Every field equal to the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import _toy, assert_same, oracle_params

pytestmark = pytest.mark.gpu
GAPS = [(-11, -2), (-32, -2)]


def _config(mode, tie, first, further):
    from pastis_gb300 import capi
    cfg = capi.config(mode, tie=tie, gap_open=first, gap_ext=further, gap_semantics=capi.GAPS_NOMINAL)
    assert capi.resolved_gaps(cfg)[:2] == (first, further)
    return cfg


@pytest.mark.parametrize("batch", [5, 131072, 131073])
@pytest.mark.parametrize("first,further", GAPS)
@pytest.mark.parametrize("tie", [0, 1, 2, 3])
@pytest.mark.parametrize("mode", [0, 1])
def test_checked_regions(native, oracle_mod, mode, tie, first, further, batch):
    """Identical W/C-rich pairs of 3500 residues pass 30000 as they are (so that the
    tagged form, the checked one and then 32-bit lanes run them); long unrelated ones
    are checked and stay; one identical pair of 1500 passes 30000 only when scaled.  The
    rest of the batch are pairs of a few residues."""
    if batch != 5 and tie in (1, 2):
        pytest.skip("two tie policies in the large batches")
    from pastis_gb300 import capi
    rng = np.random.default_rng(23)
    rich = np.frombuffer(b"WCWCWYHW", dtype=np.uint8)
    std = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", dtype=np.uint8)
    seqs = [rich[rng.integers(0, len(rich), 3500)] for _ in range(2)]
    seqs += [std[rng.integers(0, len(std), int(L))] for L in (3000, 2900, 1800, 1500)]
    seqs += [std[rng.integers(0, len(std), int(L))] for L in rng.integers(1, 12, 40)]
    ascii_ = np.concatenate(seqs)
    offs = np.cumsum([0] + [len(x) for x in seqs]).astype(np.uint64)
    pairs = np.zeros(batch, dtype=capi.PAIR_DTYPE)
    pairs["row"] = 6 + np.arange(batch) % 40
    pairs["col"] = 6 + np.arange(batch) // 40 % 40
    at = np.sort(rng.choice(batch, 5, replace=False))
    pairs["row"][at], pairs["col"][at] = [0, 1, 2, 3, 5], [0, 1, 3, 4, 5]
    pairs["rs0"][at] = pairs["cs0"][at] = [1700, 10, 5, 100, 50]
    pairs["rs1"][at] = pairs["cs1"][at] = [100, 3400, 40, 900, 1200]
    pairs["count"] = 2
    cfg = _config(mode, tie, first, further)
    O = oracle_mod
    codes = O.encode(bytes(ascii_))
    # the small pairs repeat: each one once
    _, one, inv = np.unique(pairs.view(np.uint8).reshape(batch, -1), axis=0, return_index=True, return_inverse=True)
    exp = O.batch(mode, codes, offs, codes, offs, pairs[one], oracle_params(O, cfg))[inv.ravel()]
    ctx = capi.Context(cfg)
    ctx.set_seqs(0, ascii_, offs)
    ctx.share_row_seqs()
    assert ctx.get_tuning().dp_traceback == 3
    assert_same(ctx.align(pairs), exp, pairs)
    assert (exp["score"][at[:2]] > 30000).all() and 7500 < exp["score"][at[4]] < 30000
    ctx.close()


@pytest.mark.parametrize("first,further", GAPS)
@pytest.mark.parametrize("tie", [0, 1, 2, 3])
@pytest.mark.parametrize("mode", [0, 1])
def test_half_warp_partners(native, oracle_mod, mode, tie, first, further):
    """Regions of up to 256 rows run two per warp: row counts around every multiple of
    32, partners of very different column counts, enough of them that most find one."""
    from pastis_gb300 import capi
    O = oracle_mod
    rng = np.random.default_rng(29)
    alpha = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", dtype=np.uint8)
    ms = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 129, 160, 192, 224, 255, 256, 257, 300]
    ns = [1, 3, 40, 250, 700]
    root = rng.integers(0, 20, 800)
    seqs = []
    for L in ms + ns:
        s = root[:L].copy()
        mut = rng.random(L) < 0.25
        s[mut] = rng.integers(0, 20, int(mut.sum()))
        seqs.append(alpha[s].tobytes().decode())
    w = _toy(seqs)
    npairs = 30000
    pairs = np.zeros(npairs, dtype=O.PAIR_DTYPE)
    pairs["row"] = rng.integers(0, len(ms), npairs)
    pairs["col"] = len(ms) + rng.integers(0, len(ns), npairs)
    pairs["count"] = 1
    cfg = _config(mode, tie, first, further)
    if mode == capi.MODE_XDROP:
        cfg.xdrop = 2000                               # regions up to the sequences' ends
    codes = O.encode(bytes(w.ascii))
    _, one, inv = np.unique(pairs.view(np.uint8).reshape(npairs, -1), axis=0, return_index=True, return_inverse=True)
    exp = O.batch(mode, codes, w.offs, codes, w.offs, pairs[one], oracle_params(O, cfg))[inv.ravel()]
    ctx = capi.Context(cfg)
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    assert_same(ctx.align(pairs), exp, pairs)
    ctx.close()
