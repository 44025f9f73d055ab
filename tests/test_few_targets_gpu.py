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
