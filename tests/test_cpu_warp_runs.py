"""Places where a warp's records leave as one run of consecutive slots.

The run is right only when one allocation saw all 32 lanes.  __activemask() does
not promise that (a warp may still be split after a branch, also behind
__syncwarp()), so a kernel that stores runs must not take its slots from it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "aperturerendererv3-optix-geometry_b200", "csrc")


def function(text, name):
    """The body of the function `name`, braces matched."""
    start = re.search(r"\b%s\(" % name, text).start()
    depth, i = 0, text.index("{", start)
    for k in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[i:k + 1]
    raise AssertionError(name)


def test_shading_allocates_with_the_whole_warp():
    render = open(os.path.join(CSRC, "render.cu")).read()
    stages = open(os.path.join(CSRC, "path_stages.cuh")).read()
    called = set(re.findall(r"\b(\w*alloc\w*)\(", function(render, "k_shade")))
    assert called
    for name in called:
        assert "__activemask" not in function(stages, name), name
    assert "__activemask" not in function(render, "k_shade")
