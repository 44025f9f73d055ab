"""An engine that cannot be made leaves nothing behind for the next one."""
import numpy as np
import pytest

from ermod_openacc_b200 import Engine
from ermod_openacc_b200 import systems as S
from ermod_openacc_b200.engine import ErmodError

pytestmark = pytest.mark.gpu


def test_engine_after_a_refused_one(engine_lib):
    """Energies of 10^8 insertions (410 GB) are refused for want of memory; the next engine's first
    frame must not report that."""
    w = S.make_workload(2, small=True, maxins=64)
    pos, cell = w.frame(0)
    energies = []
    for refuse in (False, True):
        if refuse:
            with pytest.raises(ErmodError, match="memory"):
                Engine(dict(w.params, maxins=10 ** 8, corrcal=0, keep_uvengy=1), w.topo, w.hist)
        eng = Engine(dict(w.params, keep_uvengy=1), w.topo, w.hist)
        assert eng.engconst(1, pos, cell) >= 0
        energies.append(eng.uvengy()[0])
        eng.close()
    assert np.array_equal(*energies)
