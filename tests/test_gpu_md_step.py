"""GPU: the MD step kernel that also finalizes its evaluation."""
import numpy as np
import pytest

import oracle_binding as ob
from gromos_nb import generators
from gromos_nb.nonbonded import Batch, Forcefield

pytestmark = pytest.mark.gpu


def start(s, **kw):
    ff = Forcefield(s)
    ff.upload_positions(s.pos)
    m = generators.masses(s)
    ff.md_init(m, generators.maxwell_velocities(m, 300.0, 3), dist_hh=generators.SPC_DHH, **kw)
    return ff


def systems():
    twin = generators.spc_water_system(700, generators.box_for_waters(700), 12, rcutp=0.8, rcutl=1.2)
    return [twin, generators.solvated_solute_system(900, 40, seed=13, single_atom_cgs=True)]


# units around a block (64) and several, with and without SETTLE, a solute, a twin range
@pytest.mark.parametrize("k,settle", [(0, True), (0, False), (1, True), (1, False)])
@pytest.mark.parametrize("steps", [1, 4, 6])
def test_forces_and_energies_of_the_last_step(k, settle, steps):
    """After md_run the context holds the last evaluation's results: those of evaluating its positions at
    the same step of the same pairlist period."""
    s = systems()[k]
    ff, ref = start(s, settle=settle), start(s, settle=settle)
    if steps > 1:
        ff.md_run(steps - 1)
        ref.md_run(steps - 1)
    st = ff.md_run(1)
    r = ff.result()
    want = ref.apply(ref.md_state()[0])  # the same step of the same period, finalized by its own kernel
    assert np.array_equal(r["forces"], want["forces"]) and np.array_equal(r["virial"], want["virial"])
    assert r["e_lj"] == want["e_lj"] and r["e_crf"] == want["e_crf"]
    assert st["e_lj"] + st["e_crf"] == pytest.approx(want["e_lj"] + want["e_crf"], rel=1e-12)
    ff.close()
    ref.close()


def test_records_written_ahead_do_not_reach_another_evaluation():
    """The step kernel writes the next step's water records; an evaluation of other positions, a graph
    replay and a batch's steps must not count their energies twice."""
    s = systems()[0]
    want = Forcefield(s).apply(s.pos)
    for graph in (False, True):
        ff = start(s)
        for _ in range(2):
            ff.apply(s.pos, graph=graph)
        ff.md_run(2)  # inside a pairlist period: the next records are written
        got = ff.apply(s.pos, force_rebuild=True, graph=graph)
        assert got["e_crf"] == want["e_crf"] and np.array_equal(got["forces"], want["forces"])
        ff.close()
    for capacity in (0, 40):  # 40: the batch's rebuild overflows, and the member runs the step on its own
        ff, b = start(s), Batch()
        ff.md_run(2)
        x = ff.md_state()[0]
        b.add(ff)
        if capacity:
            ff.set_params(list_capacity=capacity)
        b.md_run(1)
        got, want = ff.result(), Forcefield(s).apply(x)
        assert got["e_crf"] == want["e_crf"] and np.array_equal(got["forces"], want["forces"])
        assert (ff.md_stats()["rollbacks"] > 0) == (capacity > 0)
        b.close()
        ff.close()


def test_records_written_ahead_are_those_of_the_members_last_own_step():
    """A member's own steps between those of its batch: the records that they wrote ahead are of positions
    that the batch's steps leave behind."""
    s = systems()[0]
    state = []
    for fresh in (False, True):
        ff, b = start(s), Batch()
        b.add(ff)
        b.md_run(5)
        ff.md_run(2)
        b.md_run(3)  # the same recorded steps
        if fresh:
            ff.positions_device_ptr()  # the caller may write the positions: no record is kept
        ff.md_run(1)
        state.append((ff.result()["forces"], *ff.md_state()))
        b.close()
        ff.close()
    for got, want in zip(*state):
        assert np.array_equal(got, want)


def test_tiled_step_of_a_large_system():
    """More than 128 units per SM take the tiled step kernel: a last tile that is not full, solute atoms
    before the molecules, steps inside a pairlist period and across its end."""
    import torch

    waters = 128 * torch.cuda.get_device_properties(0).multi_processor_count + 467
    s = generators.solvated_solute_system(waters, 7, seed=14, single_atom_cgs=True)
    s.params.rcutp, s.params.rcutl = 0.8, 1.0
    m = generators.masses(s)
    v = generators.maxwell_velocities(m, 300.0, 3)
    ff, ref = start(s), start(s)
    ff.md_run(4)
    ref.md_run(4)
    ff.md_run(1)
    got, want = ff.result(), ref.apply(ref.md_state()[0])
    assert np.array_equal(got["forces"], want["forces"]) and got["e_crf"] == want["e_crf"]
    st = ff.md_run(1)
    x, vel = ff.md_state()
    ox, ov, so = ob.OracleForcefield(s).md_run(s.pos, v, m, 6, dist_hh=generators.SPC_DHH)
    # the bounds of the MD parity tests (FP32 pair forces over some ten steps)
    assert np.abs(x - ox).max() <= 1e-5 and np.linalg.norm(vel - ov) <= 1e-4 * np.linalg.norm(ov)
    assert abs(st["e_kin"] - so["e_kin"]) <= 1e-5 * so["e_kin"] and st["settle_failures"] == 0
    ff.close()
    ref.close()


# members of a batch below and above 16 clusters per SM (2,368): the recorded steps start their kernels
# while the predecessors end and search by blocks, or do neither
@pytest.mark.parametrize("members,waters", [(2, 700), (3, 3300)])
def test_batch_steps_equal_standalone_steps(members, waters):
    s = generators.solvated_solute_system(waters, 30, seed=15, single_atom_cgs=True)
    s.params.rcutp, s.params.rcutl = 0.8, 1.0
    alone = start(s)
    alone.md_run(7)
    want = alone.md_state()
    alone.close()
    b = Batch()
    ffs = [start(s) for _ in range(members)]
    for ff in ffs:
        b.add(ff)
    b.md_run(7)
    for ff in ffs:
        got = ff.md_state()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    b.close()
    for ff in ffs:
        ff.close()


# solvated solutes of single- and multi-atom groups, perturbed, with a twin range; a single range
@pytest.mark.parametrize("waters,solute,rcutp,kw", [(900, 30, 0.8, {"perturbed": True, "single_atom_cgs": True}),
                                                    (1200, 60, 0.8, {}), (900, 20, 1.0, {})])
def test_solute_kernels_beside_the_water_kernels(waters, solute, rcutp, kw):
    """Steps without timing events run the solute's kernels on a stream of their own: the same bits."""
    s = generators.solvated_solute_system(waters, solute, seed=16, **kw)
    s.params.rcutp, s.params.rcutl, s.params.lam = rcutp, 1.0, 0.3
    for steps in (0, 3, 5):  # the first step of a period, one inside, the first of the next
        ff, ref = start(s), start(s)
        ff.md_run(steps)
        ref.md_run(steps)
        want = ref.apply(ref.md_state()[0])
        ff.md_run(1)
        got = ff.result()
        assert np.array_equal(got["forces"], want["forces"]) and np.array_equal(got["virial"], want["virial"])
        for key in ("e_lj", "e_crf", "dhdl"):
            assert got[key] == want[key]
        ff.close()
        ref.close()
