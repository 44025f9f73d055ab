"""Large LJ tables: many atom types in one system."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine, _capi as A
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu

BOX, NSIDE = 24.9, 8


def water_energies(sites, more, maxins):
    """Energies of 512 waters with a chain solute, whose every site has an LJ type of its own, beside a
    chain molecule that brings `more` types."""
    slt, solvents, counts = S.random_chain(sites, 7), [S.water()], [NSIDE ** 3]
    pos = [S.water_box_frame(NSIDE, BOX, 5).T]
    if more:
        solvents.append(S.random_chain(more, 9))
        counts.append(1)
        pos.append(solvents[1].coords.T + BOX / 2)
    topo = S.Topology(solvents + [slt], counts + [1], [A.PT_SOLVENT] * len(solvents) + [A.PT_TEST_RIGID])
    assert topo.ljtype_max == 2 + sites + more
    prm = S.default_params(ms1max=32, maxins=maxins, corrcal=0, keep_uvengy=1)
    eng = Engine(prm, topo, dict(ecdmin=-150.0))
    assert eng.engconst(1, A.as_f32(np.concatenate(pos).ravel()), A.as_f32(np.diag([BOX] * 3).ravel())) >= 0
    u, _ = eng.uvengy()
    eng.close()
    return u[:, :NSIDE ** 3]


# 33 types: the first table outside shared memory; 142 and 168 (with 12 sites, the most that an engine
# had room for when the table had to fit a CTA's shared memory); 16, 4 and 1 lanes a molecule
@pytest.mark.parametrize("sites,more,maxins", [(30, 1, 160), (12, 128, 8), (12, 128, 40), (12, 154, 160), (30, 128, 160)])
def test_energies_do_not_depend_on_the_table(engine_lib, sites, more, maxins):
    """A water's energy is the same to the bit whatever other types the system has: the pair
    energies, the order of their sums and the solute's potential are."""
    assert np.array_equal(water_energies(sites, 0, maxins), water_energies(sites, more, maxins))
