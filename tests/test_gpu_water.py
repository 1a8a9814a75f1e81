"""GPU: the solvent kernels at their edges (clusters with members in several periodic images, long-range
pairs near half a box edge), against the FP64 oracle."""
import numpy as np
import pytest

import oracle_binding as ob
from gromos_nb import generators
from gromos_nb.nonbonded import Forcefield
from gromos_nb.system import System
from test_gpu_parity import check_pairlist, compare_eval, sorted_pairs

pytestmark = pytest.mark.gpu


# boxes little wider than twice the cutoff, and narrower: most long-range pairs near half an edge
@pytest.mark.parametrize("waters,rcutp,rcutl,width", [(343, 0.8, 1.0, 4), (343, 0.8, 1.08, 8), (400, 0.8, 1.4, 4),
                                                      (1000, 0.8, 1.4, 4)])
def test_long_range_images_in_small_boxes(waters, rcutp, rcutl, width):
    s = generators.spc_water_system(waters, generators.box_for_waters(waters), 9, rcutp=rcutp, rcutl=rcutl)
    compare_eval(s, steps=2, move=0.001, cluster_size=width)


# a seam through a layer of cells and molecules up to two boxes away: clusters with members in
# several periodic images; boxes of 2 (1,000 waters at 1.4 nm) and 3 cells per axis and more
@pytest.mark.parametrize("waters,rcutp,rcutl,layout,width", [(1000, 1.4, 1.4, 0, 0), (1000, 0.8, 1.0, 0, 8),
                                                             (3000, 0.8, 1.4, 0, 0), (3000, 1.4, 1.4, 1, 0)])
def test_lists_of_clusters_in_several_images(waters, rcutp, rcutl, layout, width):
    s = generators.spc_water_system(waters, generators.box_for_waters(waters), 6, rcutp=rcutp, rcutl=rcutl)
    rng = np.random.default_rng(waters)
    for away in (0, 2):
        x = s.pos + np.array([0.37, -0.21, 0.5]) * s.box[0]
        x = x + np.repeat(rng.integers(-away, away + 1, (waters, 3)), 3, axis=0) * s.box
        ref = ob.pairlist(System(s.topo, x, s.box, s.params), algorithm=2)
        ff = Forcefield(s, water_layout=layout, cluster_size=width)
        ff.upload_positions(x)
        ff.build_pairlist()
        for got, want in zip(ff.pairlist_lists(), ref):
            assert np.array_equal(sorted_pairs(got), sorted_pairs(want))
        ff.close()


# one block per cluster: fewer candidates than a round, several rounds and batches, lists beyond the 480
# entries that are sorted (1.9 nm), the last sizes of the kernel and the first without it (1,472 clusters)
@pytest.mark.parametrize("waters,rcutp,rcutl", [(1, 0.9, 0.9), (5, 0.8, 0.9), (130, 0.8, 0.9), (700, 1.2, 1.4),
                                                (4000, 1.9, 1.9), (4000, 0.8, 1.9), (5776, 0.8, 1.0),
                                                (5900, 0.8, 1.0)])
def test_search_by_blocks(waters, rcutp, rcutl):
    s = generators.spc_water_system(waters, max(generators.box_for_waters(waters), 2.0 * rcutl + 0.01), 8,
                                    rcutp=rcutp, rcutl=rcutl)
    check_pairlist(s)
    if waters > 100:  # a handful of waters lie outside each other's cutoff: no forces to compare
        compare_eval(s, steps=2, move=0.001)


# the search's form follows what the build before found: systems below and above 1,472 clusters, width 8,
# layout 1
@pytest.mark.parametrize("waters,layout,width", [(3000, 0, 0), (6500, 0, 0), (6500, 0, 8), (3000, 1, 0)])
def test_search_after_builds_with_and_without_several_images(waters, layout, width):
    s = generators.spc_water_system(waters, generators.box_for_waters(waters), 7, rcutp=0.8, rcutl=1.2)
    shifted = s.pos + np.array([0.37, -0.21, 0.5]) * s.box[0]
    ff = Forcefield(s, water_layout=layout, cluster_size=width)
    ref = [ob.pairlist(System(s.topo, x, s.box, s.params), algorithm=2) for x in (s.pos, shifted)]
    for k in (0, 1, 1, 0, 0):
        ff.upload_positions((s.pos, shifted)[k])
        ff.build_pairlist()
        for got, want in zip(ff.pairlist_lists(), ref[k]):
            assert np.array_equal(sorted_pairs(got), sorted_pairs(want))
    # recorded steps, before and after the first clusters in several images
    graph = Forcefield(s, water_layout=layout, cluster_size=width)
    for x in (s.pos, s.pos, s.pos, shifted, shifted, s.pos, shifted):
        a, b = ff.apply(x, force_rebuild=True), graph.apply(x, force_rebuild=True, graph=True)
        assert np.array_equal(a["forces"], b["forces"]) and a["e_crf"] == b["e_crf"]
    ff.close()
    graph.close()
