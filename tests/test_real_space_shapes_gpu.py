"""Real space in sheared cells, without a periodic box and with solvents other than 3-site water, for solutes
of one and several tiles of sites; and binning with several solvent species in solution."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine, _capi as A
from ermod_openacc_b200 import systems as S
from _helpers import bins_of, phys_uvspec

pytestmark = pytest.mark.gpu

BOX, NSIDE = 24.9, 8
SHEAR = np.array([[1.0, 0.2, 0.1], [0.0, 1.0, 0.15], [0.0, 0.0, 1.0]])


def tolerance(e, pairs):
    """FP32 coordinates (differences good to 4e-6 A here) move a contact's r^-12 by 12 4e-6 / r of it, at
    the distance r where the smallest pair (sigma 2.4 A, epsilon 0.03) has that energy; the other terms
    give 2e-5 kcal/mol for a 12-site solute and a water, growing with the root of the pairs."""
    r = 2.4 * (0.12 / np.maximum(np.abs(e), 1.0)) ** (1.0 / 12.0)
    return 48e-6 / r * np.abs(e) + 2e-5 * np.maximum(1.0, np.sqrt(pairs / 36.0))


def water4():
    w = S.water()
    return S.Species("water4", np.array([0.0, 0.52, 0.52, -1.04]), np.array([3.1536, 0.0, 0.0, 0.0]),
                     np.array([0.155, 0.0, 0.0, 0.0]), np.append(w.mass, 1e-3),
                     np.concatenate([w.coords, [[0.0], [0.15], [0.0]]], axis=1))


def placed(species, com, rng):
    """Sites [n, nsite, 3] of one molecule at every row of `com`, each turned its own way."""
    q = rng.normal(size=(len(com), 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    body = species.coords - species.coords.mean(axis=1, keepdims=True)
    return np.stack([(S._rot_from_quat(a) @ body).T for a in q]) + com[:, None, :]


def system(kind, sites, maxins, **kw):
    """(parameters, topology, mesh, sitepos, cell) of a rigid solute of `sites` sites in `kind`."""
    rng = np.random.default_rng(3)
    g = (np.arange(NSIDE) + 0.5) * (BOX / NSIDE)
    com = np.stack([a.ravel() for a in np.meshgrid(g, g, g, indexing="ij")], axis=1) + rng.normal(0.0, 0.3, (NSIDE ** 3, 3))
    com = com[rng.permutation(len(com))]
    solvents = {"water4": [(water4(), 512)], "mixed": [(S.water(), 380), (S.benzene_ring(), 60), (S.lj_site(), 72)]}.get(
        kind, [(S.water(), 512)])
    x, n0 = [], 0
    for sp, n in solvents:
        x.append(placed(sp, com[n0:n0 + n], rng).reshape(-1, 3))
        n0 += n
    x, cell = np.concatenate(x), np.eye(3) * BOX
    topo = S.Topology([sp for sp, _ in solvents] + [S.ring_recipe_solute(sites, 40 + sites)], [n for _, n in solvents] + [1],
                      [A.PT_SOLVENT] * len(solvents) + [A.PT_TEST_RIGID])
    prm = S.default_params(**dict(dict(ms1max=32, maxins=maxins, corrcal=0, keep_uvengy=1), **kw))
    if kind == "sheared":
        x, cell = x @ SHEAR.T, SHEAR * BOX
        prm.update(elecut=9.0, upljcut=9.0, lwljcut=8.0)
    if kind == "nonperiodic":
        prm.update(boxshp=A.SYS_NONPERIODIC, cltype=A.EL_COULOMB, estype=A.ES_NVT, wgtslf=0,
                   insposition=A.INSPOS_SPHERE, hostspec=1, lwreg=0.0, upreg=9.0)
    return prm, topo, dict(ecdmin=-80.0), A.as_f32(x.ravel()), A.as_f32(cell.ravel(order="F"))


# 17 and 50 sites: two and four tiles of a lane; 1, 4 and 16 lanes a molecule by the insertions (tiles of
# 16, 64 and 256 sites); 300 sites at 16 lanes: two tiles
@pytest.mark.parametrize("kind", ["sheared", "nonperiodic", "water4", "mixed"])
@pytest.mark.parametrize("sites,maxins", [(1, 8), (17, 160), (50, 160), (70, 40), (300, 8)])
def test_energies_match_oracle(oracle_mod, engine_lib, kind, sites, maxins):
    """Every per-molecule energy against the FP64 oracle on the device's own placements."""
    prm, topo, hist, pos, cell = system(kind, sites, maxins)
    eng = Engine(prm, topo, hist)
    assert eng.engconst(1, pos, cell) >= 0
    u, _ = eng.uvengy()
    ins, _ = eng.insertions()
    eng.close()
    kinds = [A.PT_SOLVENT] * (len(topo.species) - 1) + [A.PT_TEST_FLEX]
    prm_f = dict(prm, slttype=A.SLT_REFS_FLEX, insposition=A.INSPOS_NOCHANGE, insorient=A.INSROT_NOCHANGE)
    orc = oracle_mod.Oracle(prm_f, S.Topology(topo.species, topo.counts, kinds), hist, precision=8)
    assert orc.engconst(1, pos, cell, ins_conf=ins) >= 0
    uo, _ = orc.uvengy()
    tol = tolerance(uo, sites * topo.numsite[:-1].astype(float))
    assert np.all(np.abs(u - uo) <= tol), float((np.abs(u - uo) / tol).max())


# 16 lanes a molecule at 32 and 40 insertions, one at 160; batches of 32 and 64 split a target's molecules
# among other numbers of CTAs and warps than one batch does
@pytest.mark.parametrize("sites,maxins", [(12, 160), (66, 160), (66, 40), (300, 70)])
def test_energies_do_not_depend_on_the_batch(engine_lib, sites, maxins):
    res = []
    for batch in (0, 32, 64):
        prm, topo, hist, pos, cell = system("mixed", sites, maxins, ecorr_batch=batch)
        eng = Engine(prm, topo, hist)
        assert eng.engconst(1, pos, cell) >= 0
        res.append(eng.uvengy()[0])
        eng.close()
    assert np.array_equal(res[0], res[1]) and np.array_equal(res[0], res[2])


def test_solution_with_several_species(oracle_mod, engine_lib):
    """One solute, three solvent species: the bins and the species' energy sums of the wide binning CTA
    against the energies it binned."""
    prm, topo, hist, pos, cell = system("mixed", 1, 1)
    x = pos.reshape(-1, 3)
    centre = np.full(3, BOX / 2)
    slt, starts, keep = S.lj_site(), np.concatenate([[0], np.cumsum(topo.numsite[:-1])]), []
    for k in range(len(topo.numsite) - 1):                    # molecules that touch the solute are left out
        d = x[starts[k]:starts[k + 1]] - centre
        d -= BOX * np.round(d / BOX)
        keep.append(np.linalg.norm(d, axis=1).min() > 3.0)
    keep = np.array(keep)
    counts = [int(keep[a:b].sum()) for a, b in ((0, 380), (380, 440), (440, 512))]
    sites = np.concatenate([x[starts[k]:starts[k + 1]] for k in np.flatnonzero(keep)])
    topo = S.Topology([slt] + topo.species[:3], [1] + counts, [A.PT_SOLUTE] + [A.PT_SOLVENT] * 3)
    prm = S.default_params(slttype=A.SLT_SOLN, ms1max=32, maxins=1, corrcal=0, wgtslf=0, keep_uvengy=1)
    pos = A.as_f32(np.concatenate([[centre], sites]).ravel())
    eng = Engine(prm, topo, {})
    orc = oracle_mod.Oracle(prm, topo, {}, precision=8)
    assert eng.engconst(1, pos, cell) >= 0 and orc.engconst(1, pos, cell) >= 0
    u, uo = eng.uvengy()[0][0], orc.uvengy()[0][0]
    spec = phys_uvspec(topo)
    on = spec > 0
    assert np.all(np.abs(u - uo)[on] <= tolerance(uo, topo.numsite.astype(float))[on])
    for p in (1, 2, 3):
        assert eng.flceng[0, p - 1] == pytest.approx(u[spec == p].sum(), rel=1e-6, abs=1e-6)
    acc = eng.accum()
    bins = bins_of(u[None, :], eng.uvcrd, eng.uvmax, spec)[0][on]
    np.testing.assert_allclose(acc["edens"] / acc["engnorm"], np.bincount(bins, minlength=eng.ermax), rtol=1e-12)
    for p in (1, 2, 3):
        assert acc["minuv"][p] == np.float32(u[spec == p].min()) and acc["maxuv"][p] == np.float32(u[spec == p].max())
    eng.close()
