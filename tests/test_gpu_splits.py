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
    _minimized_alike((20, 40, 130, 300), 148, 149)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,few,many", [((17, 24, 32), 18, 19), ((17, 40, 64), 18, 19),
                                            ((17, 40, 96), 9, 10), ((40, 96, 97), 10, 10)])
def test_on_chip_minimizer_rules_change_no_bit(sizes, few, many):
    """Small molecules on both sides of the lines between a block each and shared units, and
    between 512 and 256 threads (148 SMs), with the same molecules in 256-thread blocks."""
    _minimized_alike(sizes, few, many)


def _minimized_alike(sizes, few, many):
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    mols = [synthetic.make_molecule(800 + k, n) for k, n in enumerate(sizes)]
    final = []
    for count, opts in ((few, {}), (many, {}), (many, dict(threads_per_block=256))):
        index = np.arange(count, dtype=np.int32) % len(mols)
        syn = sb.Synthesis(mols, topology_index=index, **opts)
        syn.set_coordinates(np.concatenate([mols[t].coords for t in index]))
        syn.minimize(total_cycles=12, sd_cycles=4, kernel=sb.MIN_PERSISTENT)
        final.append(syn.split(syn.coordinates())[:few])
        syn.close()
    for a, b, c in zip(*final):
        assert np.array_equal(a, b)
        assert np.array_equal(a, c)


@pytest.mark.gpu
def test_small_on_chip_batches_share_the_gpu():
    """Four batches of 64 small molecules on their own streams take little longer than one: with a
    512-thread block a molecule they waited for each other and took 2.1 times as long."""
    import time

    import torch
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    mol = synthetic.make_molecule(850, 20)
    index = np.zeros(64, dtype=np.int32)
    xyz = np.concatenate([mol.coords] * 64)
    syns = [sb.Synthesis([mol], topology_index=index) for _ in range(4)]
    streams = [torch.cuda.Stream() for _ in syns]

    def seconds(count):
        best = 1.0e9
        for _ in range(6):
            for syn in syns[:count]:
                syn.set_coordinates(xyz)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for syn, stream in zip(syns[:count], streams):
                syn.minimize(stream=stream.cuda_stream, total_cycles=100, sd_cycles=20,
                             kernel=sb.MIN_PERSISTENT)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best

    one, four = seconds(1), seconds(4)
    assert four <= 1.5 * one, (one, four)
    for syn in syns:
        syn.close()


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(12, 512), (300, 500)])
def test_tuned_minimizer_keeps_up_with_the_default(lo, hi):
    """128 molecules with some above 256 atoms, which the default puts in one launch: the packing
    that sb_autotune keeps was 1.3 to 1.6 times as slow while the default was no candidate."""
    import torch
    import stormm_b200 as sb
    from stormm_b200 import synthetic
    sizes = np.random.default_rng(9).integers(lo, hi + 1, size=32)
    mols = [synthetic.make_molecule(870 + k, int(n)) for k, n in enumerate(sizes)]
    index = np.arange(128, dtype=np.int32) % len(mols)
    xyz = np.concatenate([mols[t].coords for t in index])

    def milliseconds(syn):
        best = 1.0e9
        for _ in range(4):
            syn.set_coordinates(xyz)
            torch.cuda.synchronize()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            syn.minimize(total_cycles=12, sd_cycles=4, kernel=sb.MIN_PERSISTENT)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    tuned = sb.Synthesis(mols, topology_index=index)
    tuned.set_coordinates(xyz)
    tuned.autotune(sb.TUNE_MINIMIZE)
    plain = sb.Synthesis(mols, topology_index=index)
    t, d = milliseconds(tuned), milliseconds(plain)
    assert t <= 1.15 * d, (t, d)
    tuned.close()
    plain.close()


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
