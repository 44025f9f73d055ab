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


@pytest.mark.parametrize("sites", [1, 2, 3, 32, 33, 65, 130])
def test_self_energy_and_solution_frame_match_oracle(oracle_mod, engine_lib, sites):
    """One solute in solution: its sites are copied by a warp (around 32), its site pairs dealt to up
    to 512 threads (none, one, three, and past 512), one target takes the wide binning CTA.  uvengy0
    to the mesh part's FP32 (1e-6 relative + 2e-5), the energy sum to FP32 pair energies."""
    box, nside = 24.9, 8
    # sites on a compact grid, the waters that touch them moved out of its bounding sphere
    slt = S.ring_recipe_solute(sites, 7)
    m = int(np.ceil(sites ** (1.0 / 3.0)))
    grid = np.stack(np.unravel_index(np.arange(sites), (m, m, m))).astype(float) * 1.5
    slt.coords = grid - grid.mean(axis=1, keepdims=True)
    topo = S.Topology([slt, S.water()], [1, nside ** 3], [A.PT_SOLUTE, A.PT_SOLVENT])
    prm = S.default_params(slttype=A.SLT_SOLN, ms1max=32, maxins=1, corrcal=0, wgtslf=0, keep_uvengy=1)
    hist = dict(ecdmin=-80.0)
    wat = S.water_box_frame(nside, box, 11).T.reshape(-1, 3, 3) - box / 2
    r = np.linalg.norm(wat[:, 0], axis=1)
    reach = np.linalg.norm(slt.coords, axis=0).max() + 3.2
    near = r < reach
    wat[near] += (wat[near, 0] / r[near, None] * (reach - r[near, None]))[:, None, :]
    pos = A.as_f32(np.concatenate([slt.coords.T, wat.reshape(-1, 3)]).ravel() + box / 2)
    cell = A.as_f32(np.diag([box] * 3).ravel())
    eng = Engine(prm, topo, hist)
    assert eng.engconst(1, pos, cell) >= 0
    u, u0 = eng.uvengy()
    orc = oracle_mod.Oracle(prm, topo, hist, precision=8)
    assert orc.engconst(1, pos, cell) >= 0
    uo, u0o = orc.uvengy()
    assert np.allclose(u0, u0o, rtol=1e-6, atol=2e-5 * max(1.0, sites / 12.0))
    tol = np.where(np.abs(uo) < 1.0e3, 1e-5 * np.abs(uo) + 2e-5 * max(1.0, np.sqrt(sites / 12.0)), 1e-4 * np.abs(uo))
    assert np.all(np.abs(u - uo) <= tol)
    assert eng.flceng[0, 0] == pytest.approx(u.sum(), rel=1e-6)
    eng.close()
