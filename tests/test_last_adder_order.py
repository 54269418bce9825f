"""The warp that adds the last row to its part of dBias reads what other warps added: lane 0 learns of their adds from the counter, so
that its fence behind the counter and a warp barrier (a shuffle orders no memory) have to stand ahead of the other lanes' loads, as
fences and a barrier stand between the adds and the counter.  Read from the source: on a device the order holds or
not as the timing goes."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megakernel-exploration_b200", "csrc")


def test_fences_around_the_counter():
    with open(os.path.join(CSRC, "evo_bwd_halves.cuh")) as f:
        text = re.sub(r"//.*", "", f.read())
    body = text[text.index("auto count_row"):]
    body = body[:body.index("\n        };")]
    steps = re.findall(r"__threadfence|__syncwarp|__shfl_sync|atomicAdd|__ldcg|if \(lane == 0\) \{|\}", body)
    count, load = steps.index("atomicAdd"), steps.index("__ldcg")
    assert steps[:count] == ["__threadfence", "__syncwarp", "if (lane == 0) {"]
    assert steps[count + 1:steps.index("}")] == ["__threadfence"]                 # by the lane that read the counter
    assert "__syncwarp" in steps[steps.index("}"):load]
