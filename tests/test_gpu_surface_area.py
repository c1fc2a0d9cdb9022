"""The surface-area kernels at their edges: atoms with more neighbours than a warp's list holds,
point counts around the 32 and 1,024 points a warp takes at once, sphere points that are not unit
vectors, a lone atom and a system without extent along an axis; against the oracle's restatement
of STORMM's search, whose sums differ only in order (64-bit rounding, below 1e-12 relative for
the at most 1e5 addends here)."""
import copy

import numpy as np
import pytest

import oracle
from stormm_b200 import synthetic


def _points(n, scale=1.0):
    p = np.random.default_rng(n).normal(size=(n, 3))
    return scale * p / np.linalg.norm(p, axis=1)[:, None]


def _dense(natom, edge):
    """natom atoms packed into a cube: hundreds of atoms within reach of each."""
    m = copy.deepcopy(synthetic.make_molecule(5, natom))
    m.coords = np.random.default_rng(natom).uniform(0.0, edge, size=(natom, 3))
    return m


@pytest.mark.gpu
@pytest.mark.parametrize("natom,edge,npts,scale,probe", [
    (300, 6.0, 33, 1.0, 1.4), (130, 9.0, 1, 1.0, 1.4), (97, 8.0, 1025, 1.0, 1.4),
    (64, 20.0, 31, 1.0, 0.0), (90, 14.0, 272, 1.7, 2.5), (33, 12.0, 1024, 0.4, 1.4)])
def test_surface_area_edges(natom, edge, npts, scale, probe):
    import stormm_b200 as sb
    m = _dense(natom, edge)
    flat = copy.deepcopy(synthetic.make_molecule(6, 20))
    flat.coords[:, 2] = 1.0
    pair = synthetic.make_molecule(7, 2)
    batch = [m, flat, pair, m]
    pts = _points(npts, scale)
    syn = sb.Synthesis(batch)
    syn.set_coordinates(np.concatenate([q.coords for q in batch]))
    got = syn.surface_area(pts, probe_radius=probe)
    grid = syn.split(syn.coordinates())
    assert got[0] == got[3]
    assert got[1] == 0.0
    for k in (0, 2):
        ref = oracle.surface_area(grid[k], oracle.sasa_radii(batch[k]), pts, probe)
        assert abs(got[k] - ref) <= 1e-12 * max(ref, 1e-300), (k, got[k], ref)
    syn.close()
