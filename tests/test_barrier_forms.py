"""The engine's cluster barrier stands behind loops that a warp's lanes leave at
different trips, so it must not be of the `.aligned` form, whose behaviour is
undefined unless all threads of the warp execute it together."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-preprocessor-ijoc_b200", "csrc")


def test_cluster_barriers_do_not_ask_for_converged_warps():
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for form in re.findall(r'"(barrier\.cluster\.[a-z.]+);', open(path).read()):
            assert ".aligned" not in form, (os.path.basename(path), form)
            found += 1
    assert found >= 2
