"""A run's flags as the binning kernel sets them, read from the source: what sends a run from
k_curvelets to the two-kernel path (UNFIT_*) has a word of its own, and does not take that
path's shared quotients, which the certification flag decides."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "curvelet_construction_on_gpu_b200", "csrc")


def _kernel(file, name):
    with open(os.path.join(CSRC, file)) as f:
        return re.search(r"__global__ void[^;{]*\b" + name + r"\([^{]*\)\s*\{(.*?)\n\}\n", f.read(), re.S).group(1)


def test_the_certification_flag_is_the_coordinates_alone():
    body = _kernel("cvl_kernels.cuh", "k_bin_keys")
    sets = re.findall(r"[^;{}]*atomicOr\(uncertified[^;]*;", body)
    assert len(sets) == 1 and "certify_coord(x)" in sets[0] and "th" not in re.findall(r"\w+", sets[0])
    assert re.search(r"fabs\(th\).*atomicOr\(unfit, UNFIT_ANGLE\)", body)
