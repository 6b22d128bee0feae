"""The X-drop extension's division of work between threads and warps: batches on both
sides of its lines give the oracle's results, and a batch of middle size takes its share
of a larger one's time."""
import numpy as np
import pytest

from test_gpu_parity import assert_same, oracle_params

pytestmark = pytest.mark.gpu


# 12 to 576 directions a resident warp, of which 152 SMs hold 2432, are the lines; four to
# a pair
@pytest.mark.parametrize("n", [7296, 7297, 15000, 30000, 350208, 350209])
@pytest.mark.parametrize("preset", ["sw100k", "uneven10m"])
@pytest.mark.parametrize("first,further", [(None, None), (-50, -49), (-120, -100)])
def test_batch_sizes(native, oracle_mod, n, preset, first, further):
    if n > 300_000 and (preset != "sw100k" or first == -50):
        pytest.skip("the largest batches once with long directions and once without gaps")
    from pastis_gb300 import capi, synth
    w = synth.generate(preset, seed=11, nseqs=120, npairs=600, len_median=120.0, homolog_frac=0.5, len_max=2500)
    cfg = capi.config(capi.MODE_XDROP)
    if first is not None:
        cfg = capi.config(capi.MODE_XDROP, gap_open=first, gap_ext=further, gap_semantics=capi.GAPS_NOMINAL)
    at = np.arange(n) % len(w.pairs)
    O = oracle_mod
    codes = O.encode(bytes(w.ascii))
    exp = O.batch(capi.MODE_XDROP, codes, w.offs, codes, w.offs, w.pairs, oracle_params(O, cfg))[at]
    ctx = capi.Context(cfg)
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    assert_same(ctx.align(w.pairs[at]), exp, w.pairs[at])
    ctx.close()


def test_middle_batch_without_gaps(native):
    """Gap scores that do not fit into X, scored beyond the 16-bit lanes: the extension of
    20k pairs against that of 80k of the same kind takes about 0.45 of its time, 0.76 with most
    of the smaller batch's directions on warps.  By the library's own events, the best
    of several runs."""
    import torch
    from pastis_gb300 import capi, synth
    t = {}
    for n in (20_000, 80_000):
        w = synth.generate("sw100k", seed=3, nseqs=n // 5, npairs=n, len_median=250.0, homolog_frac=0.5)
        cfg = capi.config(capi.MODE_XDROP, gap_open=-120, gap_ext=-100, gap_semantics=capi.GAPS_NOMINAL)
        ctx = capi.Context(cfg)
        ctx.set_seqs(0, w.ascii, w.offs)
        ctx.share_row_seqs()
        pairs = torch.from_numpy(w.pairs.view(np.uint8).copy()).cuda()
        out = torch.zeros(n * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ms = []
        for _ in range(10):
            ctx.align_device(pairs.data_ptr(), n, out.data_ptr())
            ms.append(ctx.kernel_ms()[0])
        t[n] = min(ms[2:])
        ctx.close()
    assert t[20_000] < 0.57 * t[80_000], t
