"""Performance cases: the calls a program that uses this framework spends its
time in, at the sizes of the repository's workloads (pastis_gb300/synth.py) and
scaled-down forms of them.

A case is a plain dict.  ``op`` says which entry points run:

  align_host    Context.align: pairs in host memory, results in host memory
  align         Context.align_device: pairs and results on the device
  candidates    Context.candidates_device: the k-mer product of one block
  search        candidates, alignment and similarity triples of one block
  filter_step   Filter.predict and Filter.gradients on one mini-batch
  filtered      Filter.align_filtered: features, network, alignment of the kept

Whole numbers come back as the raw bytes of the result records.
"""
import math

import numpy as np
import torch

from pastis_gb300 import capi, synth
from pastis_gb300 import filter as pair_filter

PAIR = capi.PAIR_DTYPE.itemsize
RESULT = capi.RESULT_DTYPE.itemsize
NF, NH = 16, 64                     # the filter network: 16 -> 64 -> 64 -> 1


def _align(name, n, mode, lengths="even", gaps="called", op="align", median=250, homologs=0.5):
    return {"name": name, "op": op, "mode": mode, "pairs": n, "lengths": lengths, "gaps": gaps,
            "median": median, "homologs": homologs}


def listed():
    return [
        # one small request from a program that keeps its data on the host
        _align("xdrop_host_256", 256, "xdrop", op="align_host"),
        # the default stage (--sxa): a large batch, proteins of ordinary length
        _align("xdrop_400k", 400_000, "xdrop"),
        # the same over a protein set with a fifth of its lengths in 1000-5000
        _align("xdrop_uneven_60k", 60_000, "xdrop", lengths="uneven", median=300),
        # the gap scores taken by name (open -11, extend -2)
        _align("xdrop_nominal_20k", 20_000, "xdrop", gaps="nominal"),
        # Smith-Waterman (--sfa): the last, short batch of a run
        _align("sw_1k", 1_001, "sw"),
        # a full Smith-Waterman batch
        _align("sw_100k", 100_000, "sw"),
        # Smith-Waterman over the uneven protein set
        _align("sw_uneven_8k", 8_000, "sw", lengths="uneven", median=300),
        # Smith-Waterman with the gap scores by name: the labels the pair filter trains on
        _align("sw_nominal_40k", 40_000, "sw", gaps="nominal"),
        # candidate generation of one diagonal block of the many-to-many search
        {"name": "candidates_200k", "op": "candidates", "proteins": 200_000, "alphabet": "protein"},
        # a whole block of it: candidates, X-drop alignment, triples
        {"name": "search_60k", "op": "search", "proteins": 60_000, "alphabet": "protein"},
        # one mini-batch of the pair filter's training loop
        {"name": "filter_step_8192", "op": "filter_step", "rows": 8192},
        # a Smith-Waterman batch behind the pair filter
        _align("filtered_sw_150k", 150_000, "sw", op="filtered", homologs=0.3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["align", "align", "align", "align_host", "candidates", "search",
                     "filter_step", "filtered"])
    if op in ("candidates", "search"):
        return {"op": op, "proteins": _log(rng, 500, 150_000 if op == "candidates" else 50_000),
                "alphabet": "protein"}
    if op == "filter_step":
        return {"op": op, "rows": _log(rng, 100, 16_384)}
    c = _align("", 0, rng.choice(["xdrop", "sw"]), op=op, median=rng.randint(120, 400),
               homologs=round(rng.uniform(0.2, 0.6), 2))
    del c["name"]
    if op == "filtered":
        c["mode"], top = "sw", 100_000
    elif op == "align_host":
        top = 20_000
    else:
        kind = rng.choice(["even", "even", "uneven", "nominal"])
        if kind == "uneven":
            c["lengths"], top = "uneven", 5_000 if c["mode"] == "sw" else 40_000
        elif kind == "nominal":
            c["gaps"], top = "nominal", 20_000
        else:
            top = 80_000 if c["mode"] == "sw" else 250_000
    # longer proteins, fewer pairs: a drawn batch stays within the listed ones
    c["pairs"] = _log(rng, 50, max(100, int(top * min(1.0, (250.0 / c["median"]) ** 2))))
    return c


# ------------------------------------------------------------------ inputs
def _context(mode, gaps="called"):
    cfg = capi.config(capi.MODE_SW if mode == "sw" else capi.MODE_XDROP)
    if gaps == "nominal":
        cfg.gap_semantics = capi.GAPS_NOMINAL
    return capi.Context(cfg)


def _workload(case, seed):
    preset = "uneven10m" if case["lengths"] == "uneven" else "sw100k"
    return synth.generate(preset, seed=seed, nseqs=max(12, case["pairs"] // 5),
                          npairs=case["pairs"], len_median=float(case["median"]),
                          homolog_frac=case["homologs"])


def _network(seed):
    """He-uniform parameters in the filter's layout: W1, b1, W2, b2, w3, b3."""
    r = np.random.default_rng(seed)
    a = [np.sqrt(6.0 / NF), np.sqrt(6.0 / NH), np.sqrt(3.0 / NH)]
    return [r.uniform(-a[0], a[0], (NH, NF)), r.uniform(-0.1, 0.1, NH),
            r.uniform(-a[1], a[1], (NH, NH)), r.uniform(-0.1, 0.1, NH),
            r.uniform(-a[2], a[2], NH), np.zeros(1)]


def _batch(case, seed):
    """Features as pg_filter_features forms them (range and sign), labels of
    which a third are positive, and the training loop's weights."""
    r = np.random.default_rng(seed + 1)
    n = case["rows"]
    x = np.abs(r.normal(0.0, 0.3, (n, NF)))
    x[:, 2] = r.random(n) < 0.5
    x[:, [3, 4, 8]] *= r.choice([-1.0, 1.0], (n, 3))
    x[:, 9:11] += 0.6
    x = torch.from_numpy(x.astype(np.float32)).to(torch.bfloat16)
    y = (r.random(n) < 0.35).astype(np.float32)
    return x, y, np.where(y > 0.5, 4.0, 1.0).astype(np.float32)


def _flat32(params):
    return np.concatenate([p.ravel() for p in params]).astype(np.float32)


def prepare(case, seed):
    st = {"op": case["op"], "stream": torch.cuda.Stream()}
    op = case["op"]
    if op == "filter_step":
        f = pair_filter.Filter(0, seed=1)
        f.set_params(_flat32(_network(seed)))
        x, y, w = _batch(case, seed)
        st.update(filter=f, n=case["rows"], x=x.cuda(), y=torch.from_numpy(y).cuda(),
                  w=torch.from_numpy(w).cuda(),
                  logits=torch.empty(case["rows"], dtype=torch.float32, device="cuda"))
        return st
    if op in ("candidates", "search"):
        w = synth.generate("manytomany", seed=seed, nseqs=case["proteins"], npairs=1)
        ctx = _context("xdrop")
        ctx.set_seqs(0, w.ascii, w.offs)
        ctx.share_row_seqs()
        n = len(w.offs) - 1
        cap = int((18 + 1.2e-4 * n) * n) + 4096   # families of 2-50 and chance matches, with room
        st.update(ctx=ctx, rows=(0, n), cap=cap,
                  kc=capi.kmer_config(k=6, stride=1, prune=capi.PRUNE_EVEN_ODD, ckthr=1),
                  pairs=torch.zeros(cap * PAIR, dtype=torch.uint8, device="cuda"))
        if op == "search":
            st.update(out=torch.zeros(cap * RESULT, dtype=torch.uint8, device="cuda"),
                      tr=torch.zeros(cap, dtype=torch.int64, device="cuda"),
                      tc=torch.zeros(cap, dtype=torch.int64, device="cuda"),
                      tv=torch.zeros(cap, dtype=torch.float32, device="cuda"))
        torch.cuda.synchronize()
        return st
    w = _workload(case, seed)
    ctx = _context(case["mode"], case["gaps"])
    ctx.set_seqs(0, w.ascii, w.offs)
    ctx.share_row_seqs()
    st.update(ctx=ctx, n=len(w.pairs))
    if op == "align_host":
        st.update(pairs=w.pairs, out=np.zeros(len(w.pairs), dtype=capi.RESULT_DTYPE))
        return st
    st.update(pairs=torch.from_numpy(w.pairs.view(np.uint8).copy()).cuda(),
              out=torch.zeros(len(w.pairs) * RESULT, dtype=torch.uint8, device="cuda"))
    if op == "filtered":
        f = pair_filter.Filter(0, seed=1)
        f.set_params(_flat32(_network(seed)))
        feats = torch.empty(st["n"] * NF, dtype=torch.bfloat16, device="cuda")
        logits = torch.empty(st["n"], dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        f.features(ctx, st["pairs"].data_ptr(), st["n"], feats.data_ptr())
        f.predict(feats.data_ptr(), st["n"], logits.data_ptr())
        # keep about a half: the middle of the widest gap near the median logit
        z = np.sort(logits.cpu().numpy().astype(np.float64))
        lo, hi = int(0.4 * len(z)), max(int(0.6 * len(z)), int(0.4 * len(z)) + 2)
        z = z[lo:hi]
        g = int(np.argmax(np.diff(z)))
        st.update(filter=f, threshold=float(0.5 * (z[g] + z[g + 1])))
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------- a pass
def run(st):
    op = st["op"]
    if op == "align_host":
        return st["ctx"].align(st["pairs"], out=st["out"]).view(np.uint8)
    if op == "filter_step":
        f, n = st["filter"], st["n"]
        f.predict(st["x"].data_ptr(), n, st["logits"].data_ptr())
        grad, loss = f.gradients(st["x"].data_ptr(), st["y"].data_ptr(), st["w"].data_ptr(), n)
        return {"logits": st["logits"], "grad": grad, "loss": np.float32(loss)}
    # the program's own stream, ordered with the caller's
    cur, s = torch.cuda.current_stream(), st["stream"]
    s.wait_stream(cur)
    q = s.cuda_stream
    ctx = st["ctx"]
    if op == "align":
        ctx.align_device(st["pairs"].data_ptr(), st["n"], st["out"].data_ptr(), q)
        got = st["out"]
    elif op == "filtered":
        kept = st["filter"].align_filtered(ctx, st["threshold"], st["pairs"].data_ptr(), st["n"],
                                           st["out"].data_ptr(), q)
        got = {"kept": kept, "out": st["out"]}
    else:
        n = ctx.candidates_device(st["kc"], st["rows"], st["rows"], st["pairs"].data_ptr(),
                                  st["cap"], q)
        got = {"n": n, "pairs": st["pairs"]}     # the buffers whole: zeros past the count
        if op == "search":
            ctx.align_device(st["pairs"].data_ptr(), n, st["out"].data_ptr(), q)
            m = capi.triples_device(st["pairs"].data_ptr(), st["out"].data_ptr(), n, 0, 0,
                                    st["tr"].data_ptr(), st["tc"].data_ptr(),
                                    st["tv"].data_ptr(), q)
            got.update(triples=m, out=st["out"], rows=st["tr"], cols=st["tc"], vals=st["tv"])
    cur.wait_stream(s)
    return got


# ---------------------------------------------------------------- what it costs
def _cells(case):
    """Expected cells of the alignment matrices per pair (m x n; the X-drop
    regions are about half of that for ordinary lengths, a tenth for uneven)."""
    even = case["median"] ** 2 * math.exp(0.25)          # independent lognormal lengths, sigma 0.5
    same = case["median"] ** 2 * math.exp(0.5)           # homologs: about equal lengths
    if case["lengths"] == "uneven":
        mean = 0.8 * math.sqrt(even) + 0.2 * 3000.0
        even, same = mean * mean, 0.8 * same + 0.2 * 1.03e7
    h = case["homologs"]
    c = h * same + (1.0 - h) * even
    if case["mode"] == "xdrop":
        c *= 0.1 if case["lengths"] == "uneven" else 0.55
    return c


def work(case):
    op = case["op"]
    if op == "filter_step":
        n = case["rows"]
        macs = NF * NH + NH * NH + NH
        p = macs + 2 * NH + 1
        return {"bytes": n * (2 * NF + 12) + 4 * (2 * p + 1), "flops": 2 * n * macs * 4}
    if op in ("candidates", "search"):
        n = case["proteins"]
        res = n * 281
        chance = (res / 2.0) ** 2 / 4e7                  # k-mer matches between unrelated proteins
        found = n * 12 + 8e-5 * n * n                    # pairs with two shared k-mers
        by = res + 8 * n + found * PAIR
        ops = 2.0 * res + chance + n * 1500.0
        if op == "search":
            by += found * (RESULT + 20)
            ops += 4.0 * n * 12 * 3e4
        return {"bytes": int(by), "flops": int(ops)}
    n = case["pairs"]
    mean = case["median"] * math.exp(0.125)
    if case["lengths"] == "uneven":
        mean = 0.8 * mean + 0.2 * 3000.0
    # one add and one max per predecessor: 4 of the linear model, 7 of the affine one
    ops = n * _cells(case) * (7 if case["gaps"] == "nominal" else 4)
    if op == "filtered":
        ops *= 0.5
    return {"bytes": int(max(12, n // 5) * mean + n * (PAIR + RESULT)), "flops": int(ops)}


def exact(case, seed):
    """The network's logits, gradients and loss in 64 bits.  The other
    operations return whole numbers and record bytes."""
    if case["op"] != "filter_step":
        return None
    w1, b1, w2, b2, w3, b3 = [p.astype(np.float32).astype(np.float64) for p in _network(seed)]
    x, y, wt = _batch(case, seed)
    x = x.to(torch.float64).numpy()
    y, wt = y.astype(np.float64), wt.astype(np.float64)
    n = len(y)
    h1 = np.maximum(x @ w1.T + b1, 0.0)
    h2 = np.maximum(h1 @ w2.T + b2, 0.0)
    z = h2 @ w3 + b3[0]
    loss = np.sum(wt * (np.maximum(z, 0.0) - z * y + np.log1p(np.exp(-np.abs(z))))) / n
    dz = wt * (1.0 / (1.0 + np.exp(-z)) - y) / n
    d2 = np.outer(dz, w3) * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grad = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dz,
                           [dz.sum()]])
    return {"logits": z, "grad": grad, "loss": loss}
