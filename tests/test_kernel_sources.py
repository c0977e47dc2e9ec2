"""What a test of results cannot show, read from the kernels' sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "orb_slam2_detailed_comments_gb300",
                    "csrc")


def test_pyramid_bands_are_acquired_for_the_whole_warp():
    """Each lane acquires the bands it polls; a vote orders no memory, so a
    __syncwarp() stands between the polls and the first read of a row."""
    text = open(os.path.join(CSRC, "orbgpu_extract_kernels.cu")).read()
    body = re.search(r"bool bands_ready\(.*?\n}\n", text, flags=re.S).group(0)
    assert "ld.acquire.gpu" in body
    tail = re.sub(r"//[^\n]*", "", body[body.index("__nanosleep"):])
    assert tail.index("__syncwarp();") < tail.index("return __all_sync(")
