"""The cuFFT path's two lanes: odd chunks of 32 targets on a stream with buffers of their own."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu


def frames(eng, w, n=2):
    out = []
    for i in range(n):
        pos, cell = w.frame(i)
        assert eng.engconst(i + 1, pos, cell) >= 0
        out.append(eng.uvengy())
    return out


def same(a, b):
    return all(np.array_equal(x, y) for fa, fb in zip(a, b) for x, y in zip(fa, fb))


# 33: one target on the odd lane; 64 and 65: as many chunks on each lane, one more; 97 and 160: three and
# five chunks; batches of 64 targets: the lanes join and part again, the last batch one chunk alone
@pytest.mark.parametrize("mesh,order", [(36, 4), (48, 6)])
@pytest.mark.parametrize("maxins,batch", [(33, 0), (64, 0), (65, 0), (97, 0), (160, 64)])
def test_two_lanes_give_the_bits_of_one(engine_lib, maxins, batch, mesh, order):
    """Stage-timed runs keep one stream and one lane; every energy is the same."""
    w = S.make_workload(2, small=True, maxins=maxins)
    prm = dict(w.params, keep_uvengy=1, corrcal=0, ms1max=mesh, ms2max=mesh, ms3max=mesh, splodr=order, ecorr_batch=batch)
    res = []
    for timed in (1, 0):
        eng = Engine(dict(prm, stage_timing=timed), w.topo, w.hist)
        assert eng.paths()["spectrum_path"] == 1
        res.append(frames(eng, w, 3))
        eng.close()
    assert same(*res)


def test_no_memory_for_a_second_lane(engine_lib):
    """With room for one lane only (here 40 MB less than an engine with both uses, of which the second
    lane is 86 MB and more), the engine is made and gives the same energies."""
    import gc

    import torch
    gc.collect()                                    # engines of earlier tests give their memory back now
    w = S.make_workload(2, small=True, maxins=97)
    prm = dict(w.params, keep_uvengy=1, corrcal=0, ms1max=48, ms2max=48, ms3max=48)
    eng = Engine(prm, w.topo, w.hist)               # loads what a first engine loads
    want = frames(eng, w)
    eng.close()
    before = torch.cuda.mem_get_info()[0]
    eng = Engine(prm, w.topo, w.hist)
    used = before - torch.cuda.mem_get_info()[0]
    eng.close()
    hold = [torch.empty(torch.cuda.mem_get_info()[0] - used + (40 << 20), dtype=torch.uint8, device="cuda")]
    try:
        eng = Engine(prm, w.topo, w.hist)
        got = frames(eng, w)
        eng.close()
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    assert same(want, got)
