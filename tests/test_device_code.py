"""Rules of the device code that a compiler does not check."""
import glob
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "weldform_gb300", "csrc")


def test_no_warp_operation_takes_its_mask_from_the_lanes_that_happen_to_be_there():
    """CUDA does not promise that the lanes of __activemask() reach a later
    vote together; in a divergent loop its mask may name lanes that have left."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            assert "__activemask" not in f.read(), path
