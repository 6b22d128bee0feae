"""The bound on a block's k-mer occurrence pairs (max_products): counted exactly
before any pair is visited, so that a block of low-complexity sequences, whose
pairs number 1e11, is refused at once."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOO_MANY = "too many k-mer occurrence pairs"


def _context(seqs):
    from pastis_gb300 import capi
    ascii_ = np.frombuffer("".join(seqs).encode(), dtype=np.uint8)
    offs = np.concatenate([[0], np.cumsum([len(s) for s in seqs])]).astype(np.uint64)
    ctx = capi.Context(capi.config(capi.MODE_XDROP))
    ctx.set_seqs(0, ascii_, offs)
    ctx.share_row_seqs()
    return ctx


def _pairs(seqs, k, prune, rows, cols):
    """Occurrence pairs after the prune, k-mer by k-mer."""
    def occ(block):
        d = {}
        for i in range(*block):
            for p in range(len(seqs[i]) - k + 1):
                d.setdefault(seqs[i][p:p + k], []).append(i)
        return {m: np.array(v) for m, v in d.items()}
    r, c = occ(rows), occ(cols)
    n = 0
    for m in r.keys() & c.keys():
        R, C = r[m][:, None], c[m][None, :]
        if prune == 0:
            n += R.size * C.size
        elif prune == 1:
            odd = ((R ^ C) & 1) == 1
            n += int(((R > C) & ~odd).sum() + ((R < C) & odd).sum())
        else:
            n += int((R < C).sum())
    return n


@pytest.mark.parametrize("rows,cols", [((0, 60), (0, 60)), ((7, 50), (21, 60)), ((30, 60), (0, 30)), ((1, 28), (31, 60))])
@pytest.mark.parametrize("prune", [0, 1, 2])
def test_products_bound_is_exact(native, prune, rows, cols):
    """Accepted at exactly the block's number of pairs, refused one below it; the
    records of the accepted call are those of a call without a bound."""
    from pastis_gb300 import capi
    rng = np.random.default_rng(5)
    seqs = ["".join(rng.choice(list("ARND"), int(rng.integers(1, 90)))) for _ in range(60)]
    seqs[3] = seqs[40] = "A" * 80
    ctx = _context(seqs)
    n = _pairs(seqs, 3, prune, rows, cols)
    if n == 0:            # (the upper prune of a block below the diagonal)
        assert len(ctx.candidates(capi.kmer_config(k=3, prune=prune, max_products=1), rows, cols)) == 0
    else:
        exp = ctx.candidates(capi.kmer_config(k=3, prune=prune), rows, cols)
        got = ctx.candidates(capi.kmer_config(k=3, prune=prune, max_products=n), rows, cols)
        assert len(exp) > 0 and got.tobytes() == exp.tobytes()
        if n > 1:
            with pytest.raises(capi.PgError, match=TOO_MANY):
                ctx.candidates(capi.kmer_config(k=3, prune=prune, max_products=n - 1), rows, cols)
    ctx.close()


@pytest.mark.parametrize("prune", [0, 1, 2])
def test_low_complexity_block_is_refused_at_once(native, prune):
    """600 sequences of 600 equal residues: 1.3e11 pairs (half of them after a
    prune), above the default bound of 2^31.  The count takes microseconds; a visit
    to each pair would take minutes."""
    from pastis_gb300 import capi
    ctx = _context(["A" * 600] * 600)
    ctx.candidates(capi.kmer_config(k=6, prune=prune), (0, 2), (0, 2))      # warm
    t = time.perf_counter()
    with pytest.raises(capi.PgError, match=TOO_MANY):
        ctx.candidates(capi.kmer_config(k=6, prune=prune), (0, 600), (0, 600))
    assert time.perf_counter() - t < 1.0
    ctx.close()
