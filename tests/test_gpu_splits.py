"""Launch splits that depend on a batch's size change no result bit."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_tile_runs_change_no_bit(precision):
    """One tile a warp (a chain alone, 12,403 tiles) and runs of two (four replicas, 49,612)."""
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    m = synthetic.make_chain(77, 5000)
    alone = sb.Synthesis([m], precision=precision)
    batch = sb.Synthesis([m], topology_index=np.zeros(4, dtype=np.int32), precision=precision)
    alone.set_coordinates(m.coords)
    batch.set_coordinates(np.concatenate([m.coords] * 4))
    for syn in (alone, batch):
        syn.initialize()
        syn.evaluate()
    ea, eb = alone.energies_fixed(), batch.energies_fixed()
    fa, fb = alone.forces(), batch.split(batch.forces())
    for k in range(4):
        assert np.array_equal(ea[0], eb[k])
        assert np.array_equal(fa, fb[k])
    alone.close()
    batch.close()
