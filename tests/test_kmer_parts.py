"""Columns of the candidate generation that outgrow one block's tables (more rows,
survivors or pairs than it holds) and are done in parts of the row range, against a
sort of all occurrence pairs on the CPU."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(seq, offs):
    from pastis_gb300 import capi
    ascii_ = np.frombuffer(b"ARNDCQEGHILKMFPSTWYVBZX*J", dtype=np.uint8)[seq]
    ctx = capi.Context(capi.config(capi.MODE_XDROP))
    ctx.set_seqs(0, ascii_, offs)
    ctx.share_row_seqs()
    return ctx


def _kmers(seq, offs, block, k, cmap, base, cost):
    """codes, scores, sequence (block-relative) and offset of a block's k-mers"""
    s = np.concatenate([np.arange(int(offs[i]), max(int(offs[i]), int(offs[i + 1]) - k + 1)) for i in range(*block)])
    own = np.searchsorted(offs.astype(np.int64), s, side="right") - 1
    code = np.zeros(len(s), np.int64)
    score = np.zeros(len(s), np.int64)
    for j in range(k):
        a = cmap[seq[s + j]]
        code = code * base + a
        score += cost[a]
    return code, score, own - block[0], s - offs[own].astype(np.int64)


def _reference(seq, offs, rows, cols, k, alph=0, prune=0, ckthr=0, mosthr=-1):
    from oracle import kmer_oracle as K
    from oracle import oracle as O
    from pastis_gb300 import capi
    cmap, base, cost = K.alphabet(alph, O.blosum62())
    cmap, cost = np.array(cmap), np.array(cost)
    rc, _, rr, rp = _kmers(seq, offs, rows, k, cmap, base, cost)
    cc, cs, cr, cp = _kmers(seq, offs, cols, k, cmap, base, cost)
    order = np.argsort(rc, kind="stable")
    rc, rr, rp = rc[order], rr[order], rp[order]
    lo, hi = np.searchsorted(rc, cc, "left"), np.searchsorted(rc, cc, "right")
    n = hi - lo
    q = np.repeat(np.arange(len(cc)), n)
    j = np.arange(len(q)) - np.repeat(np.cumsum(n) - n, n) + lo[q]
    r, c = rr[j], cr[q]
    gr, gc = r + rows[0], c + cols[0]
    if prune == 1:
        odd = ((gr ^ gc) & 1) == 1
        keep = ((gr > gc) & ~odd) | ((gr < gc) & odd)
    elif prune == 2:
        keep = gr < gc
    else:
        keep = np.ones(len(r), bool)
    q, j, r, c = q[keep], j[keep], r[keep], c[keep]
    sv = (cc[q] << 32) | (rp[j] << 16) | cp[q]
    key = c * (1 << 32) + r
    o = np.lexsort((sv, key))
    key, sv, sc = key[o], sv[o], cs[q][o]
    first = np.flatnonzero(np.r_[True, key[1:] != key[:-1]]) if len(key) else np.zeros(0, np.int64)
    cnt = np.diff(np.r_[first, len(key)])
    out = np.zeros(len(first), dtype=capi.PAIR_DTYPE)
    if not len(first):
        return out
    mn, mx = sv[first], sv[first + cnt - 1]
    out["row"], out["col"] = key[first] & 0xffffffff, key[first] >> 32
    out["rs0"], out["cs0"] = (mn >> 16) & 0xffff, mn & 0xffff
    out["rs1"], out["cs1"] = np.where(cnt >= 2, (mx >> 16) & 0xffff, 0), np.where(cnt >= 2, mx & 0xffff, 0)
    out["count"] = cnt & 0xffff
    out["score"] = np.maximum.reduceat(sc, first)
    return out[(out["count"].astype(int) > ckthr) & (out["score"] > mosthr)]


def _check(seq, offs, rows, cols, k, **cfg):
    from pastis_gb300 import capi
    ctx = _context(seq, offs)
    alph = cfg.pop("alph", 0)
    exp = _reference(seq, offs, rows, cols, k, alph=alph, **cfg)
    got = ctx.candidates(capi.kmer_config(k=k, alphabet=alph, **cfg), rows, cols)
    ctx.close()
    assert len(got) == len(exp)
    for f in exp.dtype.names:
        assert np.array_equal(got[f], exp[f]), f
    return exp


def _marked(n, nrows, where, times, seed=3):
    """nrows sequences of which n hold `times` copies of one 6-mer (and sequence 0
    always), the others none of it: at the front, at the end, every third or spread."""
    rng = np.random.default_rng(seed)
    mark = np.array([3, 5, 7, 9, 11, 13])
    pick = {"front": np.arange(n), "back": np.arange(nrows - n, nrows), "third": np.arange(n) * (nrows // n),
            "spread": np.sort(rng.choice(nrows, n, replace=False))}[where]
    hold = np.zeros(nrows, bool)
    hold[pick] = True
    hold[0] = True
    parts = []
    for i in range(nrows):
        x = rng.integers(14, 20, int(rng.integers(0, 12)))      # letters outside the mark
        parts.append(np.concatenate([x] + [np.r_[mark, rng.integers(14, 20, 2)]] * times) if hold[i] else x)
    offs = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.uint64)
    return np.concatenate(parts).astype(np.uint8), offs


# 320 survivors, 1536 rows of the first table, 1000 rows a part, 1536 of its table
@pytest.mark.parametrize("n,nrows,where,times,ckthr", [
    (320, 320, "front", 1, 0), (321, 330, "front", 1, 0), (322, 2000, "third", 1, 0),
    (320, 1000, "spread", 2, 1), (321, 1000, "spread", 2, 1), (900, 4000, "back", 2, 2),
    (999, 1001, "front", 1, 0), (1000, 1000, "front", 1, 0), (1001, 3100, "third", 1, 0),
    (1535, 1535, "front", 1, 1), (1536, 1536, "front", 1, 1), (1537, 1537, "front", 1, 1),
    (1537, 40000, "spread", 2, 1), (1600, 4000, "back", 1, 0), (1791, 9000, "front", 1, 0),
    (1792, 9000, "back", 1, 0), (3000, 20000, "front", 2, 0), (3000, 20000, "back", 3, 2),
    (7001, 30000, "front", 1, 0), (6000, 6000, "front", 1, -1),
])
def test_rows_of_a_column(native, n, nrows, where, times, ckthr):
    """At the edges of both tables, rows evenly placed or all in one part (which is then
    done again in narrower ones; with several copies of the k-mer a row the room taken
    for it is more than its records, and the call is done once more)."""
    seq, offs = _marked(n, nrows, where, times)
    exp = _check(seq, offs, (0, nrows), (0, 3), 6, ckthr=ckthr)
    # column 0 holds the k-mer: times^2 pairs with every row that does
    assert int((exp["col"] == 0).sum()) >= (n - 1 if times * times > ckthr else 0)


@pytest.mark.parametrize("rows,cols", [((0, 5000), (0, 40)), ((100, 5000), (4000, 4030)), ((2500, 5000), (0, 30)),
                                       ((0, 2400), (2500, 2530))])
@pytest.mark.parametrize("prune,ckthr,mosthr,alph", [(0, 0, -1, 0), (1, 0, -1, 0), (2, 0, -1, 0), (1, 1, 14, 1), (2, 2, -1, 1)])
def test_blocks_and_prunes(native, prune, ckthr, mosthr, alph, rows, cols):
    """Short k-mers over 5000 sequences: every column meets thousands of rows."""
    rng = np.random.default_rng(23)
    lens = rng.integers(0, 70, 5000)
    lens[[0, 7, 2504, 4011]] = [900, 3000, 2, 1200]
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    seq = rng.integers(0, 22, int(offs[-1])).astype(np.uint8)
    _check(seq, offs, rows, cols, 2, prune=prune, ckthr=ckthr, mosthr=mosthr, alph=alph)


def test_many_pairs_of_few_rows(native):
    """Runs of one residue: 131072 and more pairs with a single row, a pair count of
    2^16 (0 in 16 bits: no candidate) among them."""
    lens = [700, 261, 261, 5, 1, 300, 133, 700, 6, 262]
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    seq = np.zeros(int(offs[-1]), np.uint8)
    seq[int(offs[5]) + 150] = 4
    for prune in (0, 1, 2):
        exp = _check(seq, offs, (0, 10), (0, 10), 6, prune=prune)
        if not prune:
            assert not ((exp["row"] == 1) & (exp["col"] == 2)).any()


def test_time_without_threshold(native):
    """Without a count threshold every row that shares a k-mer is a candidate: 26 times
    as many records as with ckthr = 1 here, in about twice its time (78 times when such
    columns went through an array over all rows).  5 times leaves room for a busy host."""
    import torch
    from pastis_gb300 import capi, synth
    w = synth.generate("manytomany", seed=5, nseqs=200_000, npairs=1)
    ctx = capi.Context(capi.config(capi.MODE_XDROP))
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    blk = (0, len(w.offs) - 1)
    cap = 120_000_000
    buf = torch.zeros(cap * capi.PAIR_DTYPE.itemsize, dtype=torch.uint8, device="cuda")

    def best(kc):
        ts = []
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            n = ctx.candidates_device(kc, blk, blk, buf.data_ptr(), cap)
            torch.cuda.synchronize()
            ts.append(time.perf_counter() - t)
        return n, min(ts[1:])
    n1, t1 = best(capi.kmer_config(ckthr=1, prune=capi.PRUNE_EVEN_ODD))
    n0, t0 = best(capi.kmer_config())
    ctx.close()
    assert n0 > 20 * n1
    assert t0 < 5 * t1, (t0, t1)
