"""Box copies of the pair-tile forward and input gradient: tiles that are a run of a row, whole rows and whole samples, batches,
taps and instances that end inside a box, and the shapes next to them that fall back to per-thread copies."""
import pytest

import cases
import gpu_util
from simnets_tf_b200 import abi

pytestmark = pytest.mark.gpu


def _case(name, batch, channels, height, width, instances, seed, **more):
    return cases.mex_case(name, (batch, channels, height, width), instances, (channels, 1, 1), (channels, 1, 1), softmax=True,
                          unshared_region=(2,), seed=seed, **more)


EDGES = [
    _case("run_of_a_row", 1, 33, 4, 512, 68, 701, normalize=True),
    _case("rows_of_a_sample", 2, 47, 32, 32, 132, 702, eps=0.7),
    _case("samples_end_inside", 5, 65, 16, 16, 64, 703, normalize=True),
    _case("many_samples", 9, 130, 8, 8, 140, 704, eps=-0.6),
    _case("width_4", 19, 36, 4, 4, 72, 705, normalize=True),              # (no box of a pooled dy)
    _case("maxima_unaligned", 3, 40, 8, 16, 71, 706),                     # (no box for the input gradient)
    _case("rows_of_six", 3, 40, 8, 12, 80, 707),
]


@pytest.mark.parametrize("c", EDGES, ids=lambda c: c["name"])
def test_box_edges(port, c):
    gpu_util.check_mex(port, c, flags=abi.FLAG_MEX_NO_SMALL_TILES, f64_tiebreak=True)
    gpu_util.check_mex_pooled_dy(port, c, flags=abi.FLAG_MEX_NO_SMALL_TILES)
