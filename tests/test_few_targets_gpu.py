"""Chunks of few targets against chunks of 32 lanes: the same targets, the two layouts."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(32, 32, 32), (64, 64, 64), (16, 32, 64), (64, 32, 16)])
@pytest.mark.parametrize("few", [1, 8, 33, 40, 41])
def test_few_targets_match_wide_chunks(engine_lib, mesh, few):
    """Insertion i is the same in every context, so its energies in a context of `few` insertions (a
    chunk of up to 8: one; 33 and 40: the second chunk; 41: neither) are those of a context of 64.
    Only FP64 sums are ordered differently: 1e-12 of the largest term, here a contact's energy."""
    w = S.make_workload(2, small=True, maxins=64)
    prm = dict(w.params, keep_uvengy=1, corrcal=0, ms1max=mesh[0], ms2max=mesh[1], ms3max=mesh[2])
    pos, cell = w.frame(0)
    res = []
    for m in (64, few):
        eng = Engine(dict(prm, maxins=m), w.topo, w.hist)
        assert eng.engconst(3, pos, cell) >= 0
        assert eng.paths()["spectrum_path"] in (2, 3)
        res.append(eng.uvengy())
        eng.close()
    (u, u0), (v, v0) = res
    assert np.all(np.abs(v - u[:few]) <= 1e-12 * np.abs(u[:few]) + 1e-9)
    np.testing.assert_allclose(v0, u0[:few], rtol=1e-13, atol=1e-12)


@pytest.mark.parametrize("mesh", [(128, 128, 128), (128, 16, 64), (128, 64, 32)])
@pytest.mark.parametrize("maxins", [1, 7, 9, 33])
def test_k1_128_lines_and_planes(engine_lib, mesh, maxins):
    """K1 = 128: eight targets a line CTA (one, a group less one, a group and one, a chunk and one), on
    128 x 128 planes and on the smallest.  Against the cuFFT path on the same placements: the two solves
    differ by FP32 roundings of the mesh energies (2e-5 kcal/mol here, 1e-5 relative)."""
    w = S.make_workload(2, small=True, maxins=maxins)
    prm = dict(w.params, keep_uvengy=1, corrcal=0, ms1max=mesh[0], ms2max=mesh[1], ms3max=mesh[2])
    pos, cell = w.frame(0)
    res = []
    for path in (0, 1):
        eng = Engine(dict(prm, spectrum_path=path), w.topo, w.hist)
        assert eng.engconst(2, pos, cell) >= 0
        res.append(eng.uvengy())
        eng.close()
    (u, u0), (v, v0) = res
    assert np.all(np.abs(u - v) <= 1e-5 * np.abs(v) + 2e-5)
    np.testing.assert_allclose(u0, v0, rtol=1e-6, atol=2e-5)
