"""Solvents with one long molecule (a protein, a polymer) among the waters."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine, _capi as A
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu

BOX, NSIDE = 24.9, 8


def host(atoms, at):
    """`atoms` sites of the ring's types on a compact grid of 1.5 A, centred at `at`."""
    h = S.ring_recipe_solute(atoms, 5)
    m = int(np.ceil(atoms ** (1.0 / 3.0)))
    grid = np.stack(np.unravel_index(np.arange(atoms), (m, m, m))).astype(float) * 1.5
    h.coords = grid - grid.mean(axis=1, keepdims=True) + np.asarray(at, dtype=float)[:, None]
    return h


def system(solvents, sites, maxins, **kw):
    """(parameters, topology, mesh, sitepos, cell): `solvents` = [(species, count, sites [n, 3])] and
    a rigid solute of `sites` sites.  Solvent molecules may overlap: only solute-solvent energies count."""
    topo = S.Topology([s for s, _, _ in solvents] + [S.ring_recipe_solute(sites, 40 + sites)],
                      [n for _, n, _ in solvents] + [1], [A.PT_SOLVENT] * len(solvents) + [A.PT_TEST_RIGID])
    prm = S.default_params(**dict(dict(ms1max=32, maxins=maxins, corrcal=0), **kw))
    pos = A.as_f32(np.concatenate([x for _, _, x in solvents]).ravel())
    return prm, topo, dict(ecdmin=-150.0), pos, A.as_f32(np.diag([BOX] * 3).ravel())


def waters(n=NSIDE ** 3):
    return S.water(), n, S.water_box_frame(NSIDE, BOX, 5).T[:3 * n]


def split(h):
    """The same sites as molecules of two (the ring's types alternate) and, where it is odd, the last one."""
    cut = lambda a, b: [np.asarray(getattr(h, k))[a:b] for k in ("charge", "sigma", "eps", "mass")]
    n = h.nsite // 2
    res = [(S.Species("pair", *cut(0, 2), h.coords[:, :2]), n, h.coords.T[:2 * n])]
    if h.nsite % 2:
        res.append((S.Species("last", *cut(2 * n, 2 * n + 1), h.coords[:, 2 * n:]), 1, h.coords.T[2 * n:]))
    return res


# 32 and 33 atoms: the longest molecule of a lane, the shortest of a warp; 96 and 97: one turn of a
# warp's 32 lanes (three atoms each) and one more; 16, 4 and 1 lanes a molecule by the insertions;
# solutes of one tile of sites and several; the molecule across the box's edge, so that stencils wrap;
# square meshes of the gather's own sizes and others.
@pytest.mark.parametrize("mesh", [(32, 32, 32), (64, 64, 32), (32, 64, 32)])
@pytest.mark.parametrize("atoms,sites,maxins", [(32, 17, 160), (33, 17, 160), (33, 3, 10), (96, 65, 160), (97, 65, 40),
                                                (97, 130, 10), (300, 130, 160)])
def test_energy_is_the_sum_over_its_atoms(engine_lib, atoms, sites, maxins, mesh):
    """A long molecule's energy against its atoms' as molecules of two: the same FP32 pair and mesh
    energies, summed in FP64 in another order.  39,000 pairs of 2^-53 each, 4e-12 of their absolute
    sum; the molecules of two hide terms that cancel by less than 100 times.  The waters' to the bit."""
    h = host(atoms, (1.0, BOX / 2, BOX - 1.0))
    u = []
    for solvent in ([(h, 1, h.coords.T)], split(h)):
        prm, topo, hist, pos, cell = system([waters()] + solvent, sites, maxins, keep_uvengy=1, ms1max=mesh[0],
                                            ms2max=mesh[1], ms3max=mesh[2])
        eng = Engine(prm, topo, hist)
        assert eng.engconst(1, pos, cell) >= 0
        u.append(eng.uvengy()[0])
        eng.close()
    n = NSIDE ** 3
    assert np.array_equal(u[0][:, :n], u[1][:, :n])
    one, many = u[0][:, n], u[1][:, n:]
    assert np.all(np.abs(one - many.sum(axis=1)) <= 4e-10 * np.abs(many).sum(axis=1) + 1e-10)


def test_long_molecule_costs_what_its_atoms_do(engine_lib):
    """The real-space stage with one molecule of 600 atoms against the same atoms as molecules of two:
    one lane walking the long one took 18 times as long, a warp takes 3.5 times."""
    h = host(600, (BOX / 2,) * 3)
    ms = []
    for solvent in ([(h, 1, h.coords.T)], split(h)):
        prm, topo, hist, pos, cell = system([waters()] + solvent, 130, 160, stage_timing=1)
        eng = Engine(prm, topo, hist)
        t = []
        for i in range(8):
            assert eng.engconst(i + 1, pos, cell) >= 0
            t.append(eng.timings()["real"])
        ms.append(np.median(t[3:]))
        eng.close()
    assert ms[0] <= 8.0 * ms[1], ms
