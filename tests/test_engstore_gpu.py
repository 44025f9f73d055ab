"""engstore's copies: the correlation matrix through the pinned ring, and the order of engclear."""
import numpy as np
import pytest

from ermod_openacc_b200 import Batch, Engine
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu


# ermax 350, 363, 1396 (default), 2596: below a slot (copied directly), just over one slot of
# 1 MB, past the ring's twelve slots, and several times round it
@pytest.mark.parametrize("hist", [dict(eclbin=0.5, ecfbin=0.02, ec0bin=0.002, pecore=50),
                                  dict(eclbin=0.5, ecfbin=0.02, ec0bin=0.002, pecore=63), {}, dict(ecdmin=-80.0)])
def test_engstore_is_accum_over_engnorm(engine_lib, hist):
    w = S.make_workload(2, small=True, maxins=48)
    eng = Engine(w.params, w.topo, hist)
    pos, cell = w.frame(0)
    assert eng.engconst(1, pos, cell) >= 0
    raw = eng.accum()
    out, av = eng.engstore()
    assert raw["ecorr"].any()
    assert np.array_equal(out["ecorr"], raw["ecorr"] / raw["engnorm"])
    assert np.array_equal(out["edens"], raw["edens"] / raw["engnorm"])
    assert np.array_equal(eng.accum()["ecorr"], raw["ecorr"])      # the accumulators stay as they were
    assert av[0] == raw["engnorm"] / raw["engsmpl"]
    eng.close()


def test_engclear_is_ordered_before_a_batch(engine_lib):
    """engclear returns before its work is done; a batch's frame, on another stream, comes after it."""
    ws = [S.make_workload(2, small=True, maxins=m) for m in (32, 40)]
    engines = [Engine(w.params, w.topo, w.hist) for w in ws]
    batch = Batch(engines)
    pos, cell = ws[0].frame(0)
    for e in engines:
        e.engclear()
    batch.engconst(1, pos, cell)
    want = [e.accum() for e in engines]
    for _ in range(20):
        for e in engines:
            e.engclear()
        batch.engconst(1, pos, cell)
        for e, a in zip(engines, want):
            b = e.accum()
            assert np.array_equal(a["edens"], b["edens"]) and np.array_equal(a["ecorr"], b["ecorr"])
            assert a["engsmpl"] == b["engsmpl"]
    batch.close()
