"""What a cached tuning is valid for: the build of the kernels and the scores that
choose between them, besides device and workload.  On the CPU, with fake contexts."""
import json

import numpy as np
import pytest

from test_autotune import FakeCtx


def _ctx(cfg):
    from pastis_gb300 import capi
    c = FakeCtx()
    key = capi.scoring_key(cfg)
    c.scoring_key = lambda: key
    return c


def test_scoring_keys_differ(native):
    from pastis_gb300 import capi
    sm = np.arange(625, dtype=np.int8)
    sm2 = sm.copy()
    sm2[7] += 1
    cfgs = [capi.config(capi.MODE_SW), capi.config(capi.MODE_SW, gap_semantics=capi.GAPS_NOMINAL),
            capi.config(capi.MODE_SW, gap_ext=-3), capi.config(capi.MODE_SW, xdrop=200),
            capi.config(capi.MODE_SW, flags=capi.F_XDROP_AFFINE)]
    for m in (sm, sm2):
        cfgs.append(capi.config(capi.MODE_SW))
        cfgs[-1].score_matrix = m.ctypes.data
    keys = [capi.scoring_key(c) for c in cfgs]
    assert len(set(keys)) == len(keys)
    assert capi.scoring_key(capi.config(capi.MODE_SW)) == keys[0]


@pytest.mark.parametrize("what", ["gaps", "build"])
def test_cached_pick_of_other_kernels_is_not_used(native, tmp_path, monkeypatch, what):
    """The same workload key under other gap scores, or from another build of the
    library, is searched again."""
    from pastis_gb300 import autotune, capi
    monkeypatch.setenv("PG_TUNING_CACHE", str(tmp_path / "t.json"))
    a = capi.config(capi.MODE_SW)
    b = capi.config(capi.MODE_SW, gap_semantics=capi.GAPS_NOMINAL) if what == "gaps" else a
    autotune.tune(_ctx(a), lambda: None, key="k", reps=1)
    assert autotune.tune(_ctx(a), lambda: None, key="k", reps=1)[1]["cached"]
    if what == "build":
        monkeypatch.setattr(capi, "build_key", lambda: "another")
    assert not autotune.tune(_ctx(b), lambda: None, key="k", reps=1)[1]["cached"]
    assert len(json.load(open(tmp_path / "t.json"))) == 2
