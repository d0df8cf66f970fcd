"""What the weight gate of the first GEMM orders, read from the source: several GPUs would have to meet for a run to show it."""
import os
import re

import tensornet_b200


def test_the_lane_that_loads_is_the_lane_that_has_seen_the_flags():
    path = os.path.join(os.path.dirname(tensornet_b200.__file__), "csrc", "gemm_tcgen05.cu")
    with open(path) as f:
        src = f.read()
    producer = src[src.index("TMA producer"):src.index("MMA issuer")]
    elected = producer.index("lead = elect_one()")
    gate = re.search(r"if \(p\.gate_flags != nullptr\) \{\s*if \((\w+)\) \{(.*?)fence\.proxy\.async", producer, re.S)
    assert elected < gate.start() and gate[1] == "lead" and "ld_acquire_sys_u64(p.gate_flags" in gate[2]
    loads = producer.index("tma_load_2d", gate.end())
    assert "if (lead) {" in producer[gate.end():loads]
