"""The tagged 16-bit form of the affine alignment DP at the edges of its rows per
lane, half-warp and whole-warp regions and stripes, and past the range it is proven
in, against the oracle; every field equal, so no tolerance."""
import numpy as np
import pytest

from test_gpu_parity import _toy, assert_same
from test_linear_gap import _extreme

pytestmark = pytest.mark.gpu

# rows: 32 R and 64 R rows for R up to 8 with their neighbours, two and three
# stripes, and beyond the largest provably exact side (7750 / smax); columns: odd
# counts around the two- and four-step groups, the ramps and 32-column row reads
ROWS = [1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257, 320, 321, 448, 449, 511, 512, 513, 576, 700, 1030, 1500]
COLS = [1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 251, 705, 1499]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("tie,first,further,table", [(0, -11, -2, None), (1, -5, -5, None), (2, -11, -1, None),
                                                     (3, -11, -2, None), (0, -31, -2, "extreme"),
                                                     (3, -7, -3, "extreme"), (2, -32, -2, None)])
def test_tagged_edges(native, oracle_mod, mode, tie, first, further, table):
    from pastis_gb300 import capi
    O = oracle_mod
    rng = np.random.default_rng(43)
    alpha = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", dtype=np.uint8)
    root = rng.integers(0, 20, 1600)
    seqs = []
    for k, L in enumerate(ROWS + COLS):
        s = root[:L].copy()
        mut = rng.random(L) < (0.3 if k % 3 else 0.0)     # every third one unchanged: the largest scores
        s[mut] = rng.integers(0, 20, int(mut.sum()))
        seqs.append(alpha[s].tobytes().decode())
    w = _toy(seqs)
    pairs = np.zeros(len(ROWS) * len(COLS), dtype=O.PAIR_DTYPE)
    pairs["row"] = np.repeat(np.arange(len(ROWS)), len(COLS))
    pairs["col"] = len(ROWS) + np.tile(np.arange(len(COLS)), len(ROWS))
    pairs["count"] = 1
    cfg = capi.config(mode, tie=tie, gap_open=first, gap_ext=further, gap_semantics=capi.GAPS_NOMINAL)
    if mode == capi.MODE_XDROP:
        cfg.xdrop = 5000                                  # regions up to the sequences' ends
    sm = _extreme() if table else O.blosum62()
    if table:
        cfg.score_matrix = sm.ctypes.data
    go, ge, xg = capi.resolved_gaps(cfg)
    assert (go, ge) == (first, further)
    p = O.make_params(gap_first=go, gap_ext=ge, xdrop_gap=xg, xdrop=cfg.xdrop, seed_len=cfg.seed_len,
                      seed_count=cfg.seed_count, tie=tie, flags=cfg.flags, cov_thr=cfg.cov_thr,
                      ani_thr=cfg.ani_thr, sm=sm)
    codes = O.encode(bytes(w.ascii))
    exp = O.batch(mode, codes, w.offs, codes, w.offs, pairs, p)
    ctx = capi.Context(cfg)
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    for form, rows, mb in ((3, 8, 0), (3, 8, 1), (2, 8, 0), (3, 5, 0)):
        ctx.set_tuning(dp_traceback=form, rows_max=rows, dir_arena_mb=mb)
        assert_same(ctx.align(pairs), exp, pairs)
    ctx.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("batch", [131072, 131073])
def test_walks_by_warp_and_by_thread(native, oracle_mod, mode, batch):
    """Either side of the batch size from which the tracebacks take a thread per pair
    in place of a warp."""
    from pastis_gb300 import capi
    O = oracle_mod
    rng = np.random.default_rng(47)
    alpha = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", dtype=np.uint8)
    root = rng.integers(0, 20, 80)
    seqs = []
    for L in [1, 2, 9, 31, 32, 33, 40, 57, 64, 65, 70] * 2:
        s = root[:L].copy()
        mut = rng.random(L) < 0.25
        s[mut] = rng.integers(0, 20, int(mut.sum()))
        cut = int(rng.integers(0, max(1, L // 2)))        # a gap
        seqs.append(alpha[np.delete(s, slice(cut, cut + L // 8))].tobytes().decode())
    w = _toy(seqs)
    pairs = np.zeros(121, dtype=O.PAIR_DTYPE)
    pairs["row"] = np.repeat(np.arange(11), 11)
    pairs["col"] = 11 + np.tile(np.arange(11), 11)
    pairs["count"] = 1
    cfg = capi.config(mode, gap_semantics=capi.GAPS_NOMINAL)
    if mode == capi.MODE_XDROP:
        cfg.xdrop = 500
    go, ge, xg = capi.resolved_gaps(cfg)
    p = O.make_params(gap_first=go, gap_ext=ge, xdrop_gap=xg, xdrop=cfg.xdrop, seed_len=cfg.seed_len,
                      seed_count=cfg.seed_count, tie=cfg.tie, flags=cfg.flags, cov_thr=cfg.cov_thr,
                      ani_thr=cfg.ani_thr, sm=O.blosum62())
    codes = O.encode(bytes(w.ascii))
    exp = O.batch(mode, codes, w.offs, codes, w.offs, pairs, p)
    at = np.arange(batch) % len(pairs)
    ctx = capi.Context(cfg)
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    assert_same(ctx.align(pairs[at]), exp[at], pairs[at])
    ctx.close()
