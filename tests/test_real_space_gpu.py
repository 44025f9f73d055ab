"""Real-space energies at the edges of the kernel's site tiles and lane splits."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine, _capi as A
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu


# Lanes a molecule by insertions x molecules (512 waters): 16 up to 36 insertions, 4 up to 147, then
# 1; tiles of 16 sites a lane: one site, a tile, a tile and one, and past the 64- and 256-site marks.
@pytest.mark.parametrize("sites,maxins", [(1, 8), (3, 8), (16, 8), (17, 40), (33, 150), (64, 40), (65, 8), (66, 160),
                                          (257, 8)])
def test_pair_energies_match_oracle(oracle_mod, engine_lib, sites, maxins):
    """Every per-molecule energy against the FP64 oracle on the device's own placements: soft region
    1e-5 relative + 2e-5 (the FP32 pair energies' and the mesh's rounding), contacts 1e-4 relative
    (r^-12 of FP32 coordinates)."""
    box, nside = 24.9, 8
    topo = S.Topology([S.water(), S.ring_recipe_solute(sites, 40 + sites)], [nside ** 3, 1],
                      [A.PT_SOLVENT, A.PT_TEST_RIGID])
    prm = S.default_params(ms1max=32, maxins=maxins, keep_uvengy=1, corrcal=0)
    w = S.Workload("edges", prm, topo, dict(ecdmin=-80.0), box, nside, 1, 5)
    pos, cell = w.frame(0)
    eng = Engine(prm, topo, w.hist)
    assert eng.engconst(1, pos, cell) >= 0
    u, _ = eng.uvengy()
    ins, _ = eng.insertions()
    kinds = [A.PT_SOLVENT, A.PT_TEST_FLEX]
    prm_f = dict(prm, slttype=A.SLT_REFS_FLEX, insposition=A.INSPOS_NOCHANGE, insorient=A.INSROT_NOCHANGE)
    orc = oracle_mod.Oracle(prm_f, S.Topology(topo.species, topo.counts, kinds), w.hist, precision=8)
    assert orc.engconst(1, pos, cell, ins_conf=ins) >= 0
    uo, _ = orc.uvengy()
    tol = np.where(np.abs(uo) < 1.0e3, 1e-5 * np.abs(uo) + 2e-5 * max(1.0, np.sqrt(sites / 12.0)), 1e-4 * np.abs(uo))
    assert np.all(np.abs(u - uo) <= tol), float((np.abs(u - uo) / tol).max())
    # a molecule's energy does not depend on which batch or block it falls in
    again = Engine(prm, topo, w.hist)
    assert again.engconst(1, pos, cell) >= 0
    assert np.array_equal(u, again.uvengy()[0])
    eng.close()
    again.close()
