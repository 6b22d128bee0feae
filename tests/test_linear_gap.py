"""The linear-gap alignment (first gap position cheaper than the further ones)
at the edges of its classes, lanes and stripes, against the oracle; every field
equal, so no tolerance."""
import numpy as np
import pytest

from test_gpu_parity import _toy, assert_same

pytestmark = pytest.mark.gpu

# rows: the class edges (16 R, 32 R, 64 R rows for R up to 8), a row less and a
# row more, the first stripe edges; columns: shorter than a lane's ramp, around
# the 4- and 8-step groups, past 64 (a base move) and 1024
ROWS = [1, 2, 15, 16, 17, 31, 32, 33, 64, 65, 80, 81, 96, 112, 113, 127, 128, 129, 160, 161, 192, 193,
        224, 225, 256, 257, 320, 321, 384, 385, 448, 449, 511, 512, 513, 640, 641, 1024, 1025, 1100]
COLS = [1, 2, 3, 4, 5, 7, 8, 9, 33, 61, 250, 700, 1500]


def _extreme():
    """Scores over the whole range the tagged int8 profile holds, -31 to 31."""
    rng = np.random.default_rng(5)
    s = rng.integers(-31, 12, (25, 25))
    s = np.minimum(s, s.T)
    s[np.arange(25), np.arange(25)] = rng.integers(5, 32, 25)
    s[3, 4] = s[4, 3] = -31
    s[0, 0] = 31
    return np.ascontiguousarray(s.astype(np.int8))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("tie,first,further,table", [(0, -2, -11, None), (3, -2, -11, None), (1, -1, -1000, None),
                                                     (0, -31, -32, "extreme"), (3, -3, -4, "extreme")])
def test_class_edges(native, oracle_mod, mode, tie, first, further, table):
    from pastis_gb300 import capi
    O = oracle_mod
    rng = np.random.default_rng(41)
    alpha = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", dtype=np.uint8)
    root = rng.integers(0, 20, 1600)
    seqs = []
    for L in ROWS + COLS:
        s = root[:L].copy()
        mut = rng.random(L) < 0.3
        s[mut] = rng.integers(0, 20, int(mut.sum()))
        seqs.append(alpha[s].tobytes().decode())
    w = _toy(seqs)
    pairs = np.zeros(len(ROWS) * len(COLS), dtype=O.PAIR_DTYPE)
    pairs["row"] = np.repeat(np.arange(len(ROWS)), len(COLS))
    pairs["col"] = len(ROWS) + np.tile(np.arange(len(COLS)), len(ROWS))
    pairs["count"] = 1
    cfg = capi.config(mode, tie=tie, gap_ext=first, gap_open=further)     # as PASTIS passes them
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
    for mb in (0, 1):                     # one pass, and the range halved until it fits 1 MiB
        ctx.set_tuning(dir_arena_mb=mb)
        assert_same(ctx.align(pairs), exp, pairs)
    ctx.close()
