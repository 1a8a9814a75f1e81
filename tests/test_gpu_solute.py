"""GPU: the solute pairlist search and the solute force kernels at their edges, against the FP64 oracle."""
import dataclasses

import numpy as np
import pytest

import oracle_binding as ob
from gromos_nb import generators
from gromos_nb.nonbonded import Forcefield
from gromos_nb.system import NonbondedParams, System, Topology, csr_from_lists
from test_gpu_parity import check_pairlist, compare_eval

pytestmark = pytest.mark.gpu


def linked_solute(n_waters, n_solute, seed, links, o14=0, hub=0, rcutp=0.8, rcutl=1.4, single=False):
    """A solvated solute whose charge groups share `links` random excluded atom pairs and `o14` 1-4
    pairs; `hub` charge groups exclude the first atom."""
    s = generators.solvated_solute_system(n_waters, n_solute, seed=seed, single_atom_cgs=single)
    t = s.topo
    rng = np.random.default_rng(seed + 1)
    cg = t.atom_to_cg()
    excl = [set(t.excl[t.excl_off[a]:t.excl_off[a + 1]].tolist()) for a in range(t.n_atoms)]
    f14 = [set() for _ in range(t.n_atoms)]
    pairs = [tuple(sorted(p)) for p in rng.integers(0, t.n_solute_atoms, (links + o14, 2)).tolist()]
    pairs = [p for p in pairs if cg[p[0]] != cg[p[1]]]
    first = t.cg_offsets[1:1 + hub]
    for a, b in pairs[:links] + [(0, int(b)) for b in first]:
        excl[a].add(b)
        excl[b].add(a)
    for a, b in pairs[links:]:
        if b not in excl[a]:
            f14[a].add(b)
    eo, ef = csr_from_lists([sorted(x) for x in excl], t.n_atoms)
    fo, ff = csr_from_lists([sorted(x) for x in f14], t.n_atoms)
    s.topo = dataclasses.replace(t, excl_off=eo, excl=ef, o14_off=fo, o14=ff)
    s.params.rcutp, s.params.rcutl = rcutp, rcutl
    return s


# candidate counts around the 256 of one sweep round (80: below one, 256: one exactly with the
# solute's groups, 700: several); 300 links over few groups; one group with more than the 64 masks
# that a block queues
@pytest.mark.parametrize("waters,solute,links,o14,hub,single", [
    (80, 12, 4, 3, 0, False), (226, 30, 0, 0, 0, True), (700, 60, 300, 20, 0, False),
    (900, 120, 30, 10, 80, True), (1500, 6, 0, 0, 0, False)])
def test_solute_lists_with_exclusions_between_groups(waters, solute, links, o14, hub, single):
    s = linked_solute(waters, solute, 31 + waters, links, o14, hub, single=single)
    check_pairlist(s)
    compare_eval(s, steps=2, move=0.001)


def test_excluded_terms_round_once_per_warp():
    """125 copies of an eight-atom group out of each other's reach, two energy groups: only self and
    excluded terms, whose sums in FP64 are taken to units of 2^-24 once per warp (and group pair)."""
    n, size = 125, 8
    rng = np.random.default_rng(5)
    shape, q = rng.uniform(-0.2, 0.2, (size, 3)), rng.normal(0.0, 0.4, size)
    at = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 1, 3) * 3.0 + 1.5
    eo, ex = csr_from_lists([[b for b in range(a - a % size, a - a % size + size) if b != a]
                             for a in range(n * size)], n * size)
    topo = Topology(n_solute_atoms=n * size, n_solute_cg=n,
                    cg_offsets=np.arange(0, n * size + 1, size), charge=np.tile(q, n),
                    iac=np.zeros(n * size, dtype=int), lj=np.zeros((1, 1, 4)), excl_off=eo, excl=ex,
                    o14_off=np.zeros(n * size + 1, dtype=int), o14=np.zeros(0, dtype=int),
                    egroup=np.tile([0, 1], n * size // 2), n_egroups=2)
    p = NonbondedParams(rcutp=1.0, rcutl=1.0, epsrf=61.0)
    s = System(topo=topo, pos=(shape + at).reshape(-1, 3), box=np.full(3, 15.0), params=p)
    ff = Forcefield(s)
    got = ff.apply(s.pos)
    ff.close()
    want = ob.OracleForcefield(s).apply(s.pos)
    warps = -(-n * (size + size * (size - 1) // 2) // 32)
    half = 2.0 ** -25
    assert np.abs(got["egroup_crf"] - want["egroup_crf"]).max() <= warps * half
    assert np.abs(got["virial"] - want["virial"]).max() <= warps * half
    # the terms of the copies are equal, so roundings of single terms add up: typically beyond this too
    assert abs(got["e_crf"] - want["e_crf"]) <= 3.0 * half * np.sqrt(3.0 * warps)


# solvent molecules of two kinds: the solute's entries go atom by atom with the atoms' own charges and
# types.  (Solvent pairs take the first molecule's parameters; the reference's topology knows one solvent
# only.  Its solvent loop of the short range does the same, that of the long range does not, so a twin
# range is compared on the solute's atoms.)
@pytest.mark.parametrize("waters,solute,single,rcutp", [(700, 30, True, 0.8), (700, 30, False, 0.8),
                                                        (600, 40, False, 1.2)])
def test_solvent_of_two_kinds(waters, solute, single, rcutp):
    s = generators.solvated_solute_system(waters, solute, seed=41, single_atom_cgs=single)
    s.params.rcutp, s.params.rcutl = rcutp, 1.2
    t = s.topo
    charge, iac = t.charge.copy(), t.iac.copy()
    odd = (t.n_solute_atoms + 3 * np.arange(1, waters, 2))[:, None] + np.arange(3)
    charge[odd] *= 0.8
    iac[odd[:, 0]] = iac[0]
    s.topo = dataclasses.replace(t, charge=charge, iac=iac)
    ff = Forcefield(s)
    got, want = ff.apply(s.pos)["forces"], ob.OracleForcefield(s).apply(s.pos)["forces"]
    ff.close()
    n = t.n_solute_atoms
    assert np.linalg.norm(got[:n] - want[:n]) <= 1e-5 * np.linalg.norm(want[:n])
    if rcutp == s.params.rcutl:
        compare_eval(s, steps=2, move=0.001)
