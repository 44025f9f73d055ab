"""Random insertion of larger solutes at the edges of the block shapes."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine, _capi as A
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu


# 128 threads in shared memory up to 32 sites, a warp up to 399, device memory above; 33 insertions: a
# warp and one
@pytest.mark.parametrize("sites", [32, 33, 64, 399, 400])
def test_placement_matches_oracle(oracle_mod, engine_lib, sites):
    """FP32 centre-of-mass shifts (sums over the sites) and quaternion products against FP64: the bound of
    the 12-site ring's placement test, 5e-5 A, times the growth of an FP32 sum's rounding, sqrt(sites / 12)."""
    topo = S.Topology([S.water(), S.ring_recipe_solute(sites, 40 + sites)], [512, 1],
                      [A.PT_SOLVENT, A.PT_TEST_RIGID])
    prm = S.default_params(ms1max=32, maxins=33, keep_uvengy=1, corrcal=0)
    w = S.Workload("insert", prm, topo, dict(ecdmin=-80.0), 24.9, 8, 1, 5)
    pos, cell = w.frame(0)
    eng, orc = Engine(prm, topo, w.hist), oracle_mod.Oracle(prm, topo, w.hist, precision=8)
    assert eng.engconst(3, pos, cell) >= 0
    assert orc.engconst(3, pos, cell) >= 0
    ins, wts = eng.insertions()
    np.testing.assert_allclose(ins, np.asarray(orc.insertions()).reshape(ins.shape), atol=5e-5 * np.sqrt(sites / 12.0))
    assert np.all(wts == 1.0)
    eng.close()
