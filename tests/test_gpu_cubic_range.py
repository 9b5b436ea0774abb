"""The FP64 overrelaxation root where the cubic's slope is near the end of
FP32's range and beyond it: the FP32 start and the FP32 reciprocal of the slope
are then no good, and the root has to come from the FP64 formula.  The triplet's
proposals against the long-double root, within the same 1e-13 of their length as
for ordinary fields (test_gpu_cubic.py): the root's condition does not depend on
the scale."""
import pytest

from test_gpu_cubic import test_triplet_proposals as proposals_match

pytestmark = pytest.mark.gpu


# slopes of about 1e36, 1e38, 1e39, 1e41 and 1e49
@pytest.mark.parametrize("scale", [3e18, 3e19, 1e20, 1e21, 1e25])
def test_slopes_beyond_fp32(scale):
    proposals_match(scale, 0.1)
