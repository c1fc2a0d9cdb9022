"""The packed tile walks at the sizes where their lanes run out: last blocks of 1, 15, 16, 17, 31
and 32 atoms, alone and behind full blocks, on the fused and the tiled path, and the list of
overlapping pairs beyond its 128 entries.  Energies and forces are held to the tolerances of
fixtures.py.

Contracted molecules (coordinates scaled until most pairs of a tile overlap) are compared by psi,
the descreening sums: every pair adds with the same sign, a pair's FP32 evaluation errs by some
3e-7 of its closed form's terms (about a dozen roundings of 6e-8), the terms are at most about
twelve times the integral they cancel to, and the workspace is read on a 2^-24 grid (plus a 2^-30
rounding per partner), hence 4e-6 |psi| + 1e-7."""
import copy

import numpy as np
import pytest

import oracle
import stormm_b200 as sb
from fixtures import FORCE_TOL, check_energies, oracle_magnitudes, rms_rel
from stormm_b200 import synthetic

pytestmark = pytest.mark.gpu

SIZES = [2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80, 81, 112, 129]


@pytest.mark.parametrize("route", ["fused", "tiled"])
def test_block_edges_match_the_oracle(route):
    mols = [synthetic.make_molecule(4000 + n, n) for n in SIZES]
    opts = dict(tiled_above_atoms=32) if route == "tiled" else {}
    syn = sb.Synthesis(mols, **opts)
    syn.set_coordinates(np.concatenate([m.coords for m in mols]))
    syn.initialize()
    syn.evaluate()
    e, f = syn.energy_terms(), syn.split(syn.forces())
    syn.initialize()
    syn.evaluate(force=False)
    alone = syn.energy_terms()
    for k, m in enumerate(mols):
        ref = oracle.from_molecule(m).evaluate(m.coords)
        rss = oracle_magnitudes(m)
        check_energies(e[k], ref["energies"], rss, (route, m.natom))
        check_energies(alone[k], ref["energies"], rss, (route, m.natom, "energy only"))
        assert rms_rel(f[k], ref["forces"]) <= FORCE_TOL, (route, m.natom)
    syn.close()


@pytest.mark.parametrize("route", ["fused", "tiled", "fp64"])
@pytest.mark.parametrize("natom,scale", [(16, 0.2), (40, 0.25), (64, 0.15), (97, 0.3)])
def test_overlapping_pairs_beyond_the_list(route, natom, scale):
    m = copy.deepcopy(synthetic.make_molecule(4100 + natom, natom))
    m.coords = m.coords * scale
    opts = {"fused": {}, "tiled": dict(tiled_above_atoms=32), "fp64": dict(precision=1)}[route]
    ref = oracle.from_molecule(m).evaluate(m.coords)
    syn = sb.Synthesis([m], **opts)
    syn.set_coordinates(m.coords)
    for force in (True, False):
        syn.initialize()
        syn.evaluate(terms=sb.TERM_GB, force=force)
        psi = syn.gb_workspace()[0]
        err = np.abs(psi - ref["psi"])
        assert np.all(err <= 4.0e-6 * np.abs(ref["psi"]) + 1.0e-7), (force, err.max())
    syn.close()


@pytest.mark.parametrize("grow", [1.0, 2.2])
@pytest.mark.parametrize("gap", [5.0, 9.9, 10.04, 10.06, 13.0, 17.0])
def test_plain_tiles_match_the_oracle(gap, grow):
    """Two blocks of atoms `gap` apart, on both sides of the distance from which the tiled path
    leaves out what only near pairs need (10 A, or four times the largest screened radius)."""
    m = copy.deepcopy(synthetic.make_molecule(4200, 96))
    rng = np.random.default_rng(7)
    # three compact clusters in a row along x, one per block of 32 atoms
    xyz = synthetic.make_molecule(4201, 32).coords
    xyz = xyz - xyz.mean(axis=0)
    width = np.ptp(xyz[:, 0])
    m.coords = np.concatenate([xyz + [k * (width + gap), 0.0, 0.0] for k in range(3)])
    m.coords = m.coords + rng.normal(0.0, 1.0e-3, size=m.coords.shape)
    m.pb_radii = m.pb_radii * grow
    m.excl12 = [set() for _ in range(96)]
    m.excl13 = [set() for _ in range(96)]
    m.excl14 = [set() for _ in range(96)]
    if gap < 6.0:
        m.excl12[3] = {70}
        m.excl12[70] = {3}
    terms = sb.TERM_NONBONDED | sb.TERM_GB
    ref = oracle.from_molecule(m).evaluate(m.coords, terms=6)
    syn = sb.Synthesis([m], tiled_above_atoms=32)
    syn.set_coordinates(m.coords)
    syn.initialize()
    syn.evaluate(terms=terms)
    check_energies(syn.energy_terms()[0], ref["energies"], oracle_magnitudes(m), (gap, grow))
    assert rms_rel(syn.forces(), ref["forces"]) <= FORCE_TOL, (gap, grow)
    syn.close()


def _excluded_pair(m):
    """Two atoms of the first block whose pair is excluded (bonded), of the largest screened
    radius: the one whose descreening grows fastest at short range."""
    s = np.asarray(m.gb_screen) * (np.asarray(m.pb_radii) - 0.09)
    pairs = [(i, j) for i in range(min(32, m.natom)) for j in m.excl12[i] if i < j < 32]
    return max(pairs, key=lambda p: s[list(p)].max())


@pytest.mark.parametrize("route", ["fused", "tiled", "fp64"])
@pytest.mark.parametrize("apart", [0.02, 0.01, 0.005, 0.001])
@pytest.mark.parametrize("natom", [40, 70])
@pytest.mark.parametrize("clash", [False, True])
def test_nearly_coincident_atoms_match_the_oracle(route, apart, natom, clash):
    """One pair far inside the other's sphere in an otherwise ordinary molecule, excluded or, with
    softened cores, not.  The closed form's terms are about 1 / (2 apart) there, so an FP32
    evaluation of them (a dozen roundings of 6e-8) errs by up to 3.6e-7 / apart in psi, which
    moves a radius R by R dpsi, and the other atoms' forces by as much for each of the two atoms
    (R is below 5 A)."""
    m = copy.deepcopy(synthetic.make_molecule(4300 + natom, natom))
    a, b = _excluded_pair(m)
    m.coords[b] = m.coords[a] + apart * np.array([0.6, 0.0, 0.8])
    if clash:
        for sets in (m.excl12, m.excl13, m.excl14):
            sets[a].discard(b)
            sets[b].discard(a)
    # the coordinates as the fixed-point grid holds them
    m.coords = np.rint(m.coords * 2.0 ** 32) * 2.0 ** -32
    soft = dict(clash_distance=0.2, clash_ratio=0.5) if clash else {}
    terms = sb.TERM_NONBONDED | sb.TERM_GB
    ref = oracle.from_molecule(m).evaluate(m.coords, terms=terms, **soft)
    opts = {"fused": {}, "tiled": dict(tiled_above_atoms=32), "fp64": dict(precision=1)}[route]
    syn = sb.Synthesis([m], **opts)
    syn.set_coordinates(m.coords)
    bound = 3.6e-7 / apart
    others = np.setdiff1d(np.arange(natom), [a, b])
    for force in (True, False):
        syn.initialize()
        if clash:
            syn.evaluate_clash(0.2, 0.5, terms=terms, force=force)
        else:
            syn.evaluate(terms=terms, force=force)
        err = np.abs(syn.gb_workspace()[0] - ref["psi"])
        assert np.all(err[others] <= 4.0e-6 * np.abs(ref["psi"][others]) + 1.0e-7), force
        assert np.all(err[[a, b]] <= 4.0e-6 * np.abs(ref["psi"][[a, b]]) + bound), (force, err)
        if force:
            f = syn.forces()
            assert rms_rel(f[others], ref["forces"][others]) <= FORCE_TOL + 10.0 * bound
    syn.close()


@pytest.mark.parametrize("route", ["fused", "tiled"])
@pytest.mark.parametrize("force", [True, False])
def test_coincident_atoms_descreen_nothing_of_each_other(route, force):
    """At r = 0 the pair adds nothing to either sum, as if each met the other far away (at 500 A
    it adds less than 1e-7)."""
    m = copy.deepcopy(synthetic.make_molecule(4370, 70))
    a, b = _excluded_pair(m)
    oracle_psi = np.zeros(70)
    for keep, gone in ((a, b), (b, a)):
        m.coords[b] = m.coords[a]
        x = m.coords.copy()
        x[gone] += [500.0, 0.0, 0.0]
        oracle_psi[keep] = oracle.from_molecule(m).evaluate(x)["psi"][keep]
    opts = dict(tiled_above_atoms=32) if route == "tiled" else {}
    syn = sb.Synthesis([m], **opts)
    syn.set_coordinates(m.coords)
    syn.initialize()
    syn.evaluate(terms=sb.TERM_GB, force=force)
    psi = syn.gb_workspace()[0][[a, b]]
    ref = oracle_psi[[a, b]]
    assert np.all(np.abs(psi - ref) <= 4.0e-6 * np.abs(ref) + 2.0e-7), (psi, ref)
    syn.close()
