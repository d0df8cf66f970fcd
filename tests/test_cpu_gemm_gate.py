"""What the weight gate of the first GEMM orders, read from the source: several GPUs would have to meet for a run to show it."""
import os
import re

import tensornet_b200


def test_the_lane_that_loads_is_ordered_behind_the_flags():
    """One lane polls; a barrier of the warp, which orders memory as a shuffle does not, and the proxy fence of every lane follow
    before any lane may load a tile."""
    path = os.path.join(os.path.dirname(tensornet_b200.__file__), "csrc", "gemm_tcgen05.cu")
    with open(path) as f:
        src = re.sub(r"//.*", "", f.read())
    producer = src[src.index("const int first_turn"):src.index("tma_load_2d(")]
    gate = producer[producer.index("if (p.gate_flags != nullptr) {"):producer.index("elect_one()")]
    poll, behind = gate.split("__syncwarp();")
    assert "ld_acquire_sys_u64(p.gate_flags" in poll and "fence.proxy.async" in behind
    assert poll.count("{") - poll.count("}") == 1                     # the barrier is for all lanes, not in the branch of the polling one
