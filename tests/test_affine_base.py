"""The tagged affine DP on a moving base (regions past the range of the scaled 16-bit
values): every rows-per-lane instance, stripes, short rows against very long columns,
scores far past 16 bits and maxima that tie, against the oracle; every field equal."""
import numpy as np
import pytest

from test_gpu_parity import _toy, assert_same
from test_linear_gap import _extreme

pytestmark = pytest.mark.gpu
ALPHA = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", dtype=np.uint8)


def _run(O, mode, seqs, rows, cols, tie, first, further, sm, tunings):
    from pastis_gb300 import capi
    w = _toy([ALPHA[s].tobytes().decode() for s in seqs])
    pairs = np.zeros(len(rows), dtype=O.PAIR_DTYPE)
    pairs["row"], pairs["col"], pairs["count"] = rows, cols, 1
    cfg = capi.config(mode, tie=tie, gap_open=first, gap_ext=further, gap_semantics=capi.GAPS_NOMINAL)
    if mode == capi.MODE_XDROP:
        cfg.xdrop = 1 << 20                           # regions up to the sequences' ends
    cfg.score_matrix = sm.ctypes.data
    go, ge, xg = capi.resolved_gaps(cfg)
    p = O.make_params(gap_first=go, gap_ext=ge, xdrop_gap=xg, xdrop=cfg.xdrop, seed_len=cfg.seed_len,
                      seed_count=cfg.seed_count, tie=tie, flags=cfg.flags, cov_thr=cfg.cov_thr,
                      ani_thr=cfg.ani_thr, sm=sm)
    codes = O.encode(bytes(w.ascii))
    exp = O.batch(mode, codes, w.offs, codes, w.offs, pairs, p)
    ctx = capi.Context(cfg)
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    for t in tunings:
        ctx.set_tuning(**t)
        assert_same(ctx.align(pairs), exp, pairs)
    ctx.close()
    return exp


def _mutant(rng, root, L, rate):
    s = root[:L].copy()
    mut = rng.random(L) < rate
    s[mut] = rng.integers(0, 20, int(mut.sum()))
    return s


# largest score 31: scaled values are provably in range up to 250 rows or columns, and
# the common pass tries up to 500
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("tie,first,further", [(0, -11, -2), (1, -31, -31), (2, -7, -1), (3, -31, -3)])
def test_rows_and_stripes(native, oracle_mod, mode, tie, first, further):
    rng = np.random.default_rng(61)
    root = rng.integers(0, 20, 2300)
    rows = [501, 512, 513, 575, 576, 577, 640, 641, 703, 769, 1023, 1024, 1025, 1500, 2100]
    cols = [501, 502, 511, 512, 513, 543, 544, 545, 999, 2003]
    seqs = [_mutant(rng, root, L, 0.3 if k % 3 else 0.0) for k, L in enumerate(rows + cols)]
    r, c = np.repeat(np.arange(len(rows)), len(cols)), len(rows) + np.tile(np.arange(len(cols)), len(rows))
    tunings = [dict(rows_max=k) for k in range(8, 0, -1)] + [dict(rows_max=8, dp_traceback=2), dict(dp_traceback=3, dir_arena_mb=1)]
    exp = _run(oracle_mod, mode, seqs, r, c, tie, first, further, _extreme(), tunings)
    assert exp["score"].max() > 10000


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("tie", [0, 3])
def test_short_against_long(native, oracle_mod, mode, tie):
    """One to 70 rows against 3650 to 9000 columns: the border row alone leaves the range
    of the scaled values (from m + n = 3719 on, with a further gap of -2)."""
    rng = np.random.default_rng(67)
    root = rng.integers(0, 20, 9000)
    rows = [1, 2, 15, 16, 17, 31, 33, 64, 70]
    cols = [3650, 3718, 3719, 4001, 9000]
    seqs = [_mutant(rng, root[200:], L, 0.2) for L in rows] + [_mutant(rng, root, L, 0.1) for L in cols]
    r, c = np.repeat(np.arange(len(rows)), len(cols)), len(rows) + np.tile(np.arange(len(cols)), len(rows))
    O = oracle_mod
    _run(O, mode, seqs, np.concatenate([r, c]), np.concatenate([c, r]), tie, -11, -2, O.blosum62(),
         [dict(), dict(rows_max=3), dict(rows_max=1)])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("tie", [0, 1, 2, 3])
def test_large_scores_and_ties(native, oracle_mod, mode, tie):
    """Identical pairs of 7000 (score past 38000, four times that scaled), a homologous
    block between unrelated ends (a score that climbs and falls again), a deletion of 900
    residues, and a motif repeated between mismatches (the same maximum at many cells)."""
    rng = np.random.default_rng(71)
    a = rng.integers(0, 20, 7000)
    block = rng.integers(0, 20, 2600)

    def noise(n):
        return rng.integers(0, 20, n)
    motif = np.concatenate([rng.integers(0, 20, 40)])
    rep1 = np.concatenate([np.concatenate([motif, np.full(60, 18)]) for _ in range(18)])     # W between
    rep2 = np.concatenate([np.concatenate([motif, np.full(55, 2)]) for _ in range(17)])      # D between
    seqs = [a, a.copy(), np.concatenate([noise(700), block, noise(1500)]),
            np.concatenate([noise(1900), _mutant(rng, block, 2600, 0.1), noise(300)]),
            np.concatenate([a[:3000], a[3900:]]), rep1, rep2]
    r, c = [0, 2, 0, 4, 5, 6, 5, 3], [1, 3, 4, 1, 6, 5, 5, 2]
    O = oracle_mod
    exp = _run(O, mode, seqs, r, c, tie, -11, -1, O.blosum62(), [dict(), dict(rows_max=5)])
    assert exp["score"][0] > 33000


def test_long_homologs_are_done_once(native):
    """A Smith-Waterman batch whose longest pairs are homologs of thousands of residues:
    with gaps of -11 / -2 (tagged) it takes 0.8 of the time it takes with -32 / -2 (the
    untagged forms), 1.47 when such pairs ran in both.  The best of several runs."""
    import torch
    from pastis_gb300 import capi, synth
    w = synth.generate("uneven10m", seed=3, nseqs=200, npairs=1000, len_median=300.0, homolog_frac=0.5)
    pairs = torch.from_numpy(w.pairs.view(np.uint8).copy()).cuda()
    out = torch.zeros(len(w.pairs) * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    t = []
    for first in (-11, -32):
        ctx = capi.Context(capi.config(capi.MODE_SW, gap_open=first, gap_ext=-2, gap_semantics=capi.GAPS_NOMINAL))
        ctx.set_seqs(0, w.ascii, w.offs)
        ctx.share_row_seqs()
        torch.cuda.synchronize()
        ms = []
        for _ in range(6):
            ctx.align_device(pairs.data_ptr(), len(w.pairs), out.data_ptr())
            ms.append(sum(ctx.kernel_ms()))
        t.append(min(ms[1:]))
        ctx.close()
    assert t[0] < 1.1 * t[1], t
