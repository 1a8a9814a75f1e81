"""GPU: the solvent kernels at their edges (lists shared by several warps, the search's buffers, clusters in
several periodic images, long-range pairs near half a box edge), against the FP64 oracle."""
import numpy as np
import pytest

from gromos_nb import generators
from test_gpu_parity import check_pairlist, compare_eval

pytestmark = pytest.mark.gpu


# boxes little wider than twice the cutoff, and narrower: most long-range pairs near half an edge
@pytest.mark.parametrize("waters,rcutp,rcutl,width", [(343, 0.8, 1.0, 4), (343, 0.8, 1.08, 8), (400, 0.8, 1.4, 4),
                                                      (1000, 0.8, 1.4, 4)])
def test_long_range_images_in_small_boxes(waters, rcutp, rcutl, width):
    s = generators.spc_water_system(waters, generators.box_for_waters(waters), 9, rcutp=rcutp, rcutl=rcutl)
    compare_eval(s, steps=2, move=0.001, cluster_size=width)
