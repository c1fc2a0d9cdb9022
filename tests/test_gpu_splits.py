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


@pytest.mark.gpu
@pytest.mark.parametrize("count,threads", [(296, 512), (300, 256), (592, 256), (760, 128),
                                           (2400, 128)])
def test_packing_and_block_size_rules_change_no_bit(count, threads):
    """The default packing and block size of batches of small molecules on both sides of each
    line (148 SMs), against one molecule a unit in 256-thread blocks."""
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    mols = [synthetic.make_molecule(700 + k, n) for k, n in enumerate((17, 24, 33, 47, 64, 96))]
    index = np.arange(count, dtype=np.int32) % len(mols)
    xyz = np.concatenate([mols[t].coords for t in index])
    syns = [sb.Synthesis(mols, topology_index=index),
            sb.Synthesis(mols, topology_index=index, threads_per_block=256, max_tiles_per_unit=1)]
    assert syns[0].launch_info()["threads"] == threads
    out = []
    for syn in syns:
        syn.set_coordinates(xyz)
        syn.initialize()
        syn.evaluate()
        out.append((syn.energies_fixed(), syn.forces_fixed()[0]))
        syn.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.gpu
def test_on_chip_minimizer_block_size_changes_no_bit():
    """148 molecules take a 512-thread block each, 149 share units of 256-thread blocks."""
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    mols = [synthetic.make_molecule(800 + k, n) for k, n in enumerate((20, 40, 130, 300))]
    final = []
    for count in (148, 149):
        index = np.arange(count, dtype=np.int32) % len(mols)
        syn = sb.Synthesis(mols, topology_index=index)
        syn.set_coordinates(np.concatenate([mols[t].coords for t in index]))
        syn.minimize(total_cycles=12, sd_cycles=4, kernel=sb.MIN_PERSISTENT)
        final.append(syn.split(syn.coordinates())[:148])
        syn.close()
    for a, b in zip(*final):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_widest_blocks_change_no_bit():
    """148 molecules of sixteen tiles and more take 1,024-thread blocks, 149 of them 512."""
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    mols = [synthetic.make_molecule(900 + k, n) for k, n in enumerate((193, 200, 224, 256))]
    out = []
    for count, threads in ((148, 1024), (149, 512)):
        index = np.arange(count, dtype=np.int32) % len(mols)
        syn = sb.Synthesis(mols, topology_index=index)
        assert syn.launch_info()["threads"] == threads
        syn.set_coordinates(np.concatenate([mols[t].coords for t in index]))
        syn.initialize()
        syn.evaluate()
        out.append((syn.energies_fixed()[:148], syn.split(syn.forces())[:148]))
        syn.close()
    assert np.array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
