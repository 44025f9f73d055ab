"""Direct site sums of square planes at the edges of the tensor-core tiles and of the plane pairs."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine, _capi as A
from ermod_openacc_b200 import systems as S

pytestmark = pytest.mark.gpu


# tiles of 16 sites; 32 targets a chunk: an odd and an even number of planes share the pairs, whole chunks,
# an odd last one, one target more than a chunk
@pytest.mark.parametrize("mesh,sites", [(64, 1), (64, 3), (64, 16), (64, 17), (64, 32), (128, 1), (128, 15), (128, 16),
                                        (128, 17), (128, 33), (128, 60)])
@pytest.mark.parametrize("maxins,box", [(33, 24.9), (9, 31.0), (64, 28.0)])
def test_plane_sums_match_cufft_path(engine_lib, mesh, sites, maxins, box):
    """The fused solve against spreading and cuFFT on the same placements: the mesh energies differ by
    FP32 roundings (2e-5 kcal/mol for 12 sites, growing as the root of their number, 1e-5 relative)."""
    nside = 8
    topo = S.Topology([S.water(), S.ring_recipe_solute(sites, 40 + sites)], [nside ** 3, 1],
                      [A.PT_SOLVENT, A.PT_TEST_RIGID])
    prm = S.default_params(ms1max=mesh, ms2max=mesh, ms3max=mesh, maxins=maxins, keep_uvengy=1, corrcal=0)
    w = S.Workload("planes", prm, topo, dict(ecdmin=-80.0), box, nside, 1, 5)
    pos, cell = w.frame(0)
    res = []
    for path in (0, 1):
        eng = Engine(dict(prm, spectrum_path=path), topo, w.hist)
        assert eng.engconst(1, pos, cell) >= 0
        res.append(eng.uvengy())
        eng.close()
    (u, u0), (v, v0) = res
    atol = 2e-5 * max(1.0, np.sqrt(sites / 12.0))
    assert np.all(np.abs(u - v) <= 1e-5 * np.abs(v) + atol)
    np.testing.assert_allclose(u0, v0, rtol=1e-6, atol=atol)


@pytest.mark.parametrize("mesh", [(64, 64, 64), (16, 16, 16), (32, 64, 16), (16, 64, 128), (16, 128, 64)])
@pytest.mark.parametrize("sites,order", [(33, 4), (65, 6), (200, 4), (90, 8)])
def test_plane_spreading_matches_cufft_path(engine_lib, mesh, sites, order):
    """Solutes past the direct sums' limit, spread on the planes in two 32-bit words a sum: planes with fewer
    threads than stencil points, planes of 8192 points.  Same bounds."""
    topo = S.Topology([S.water(), S.ring_recipe_solute(sites, 40 + sites)], [512, 1],
                      [A.PT_SOLVENT, A.PT_TEST_RIGID])
    prm = S.default_params(ms1max=mesh[0], ms2max=mesh[1], ms3max=mesh[2], splodr=order, maxins=9, keep_uvengy=1,
                           corrcal=0)
    w = S.Workload("planes", prm, topo, dict(ecdmin=-80.0), 24.9, 8, 1, 5)
    pos, cell = w.frame(0)
    res = []
    for path in (0, 1):
        eng = Engine(dict(prm, spectrum_path=path), topo, w.hist)
        assert eng.engconst(1, pos, cell) >= 0
        res.append(eng.uvengy())
        eng.close()
    (u, u0), (v, v0) = res
    atol = 2e-5 * max(1.0, np.sqrt(sites / 12.0))
    assert np.all(np.abs(u - v) <= 1e-5 * np.abs(v) + atol)
    np.testing.assert_allclose(u0, v0, rtol=1e-6, atol=atol)
