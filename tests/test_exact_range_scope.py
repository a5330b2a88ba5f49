"""The exact DeepSeek mode notes activations whose products may round; what one call saw must not steer the next.  The flag
changes no result, so this reads the host code: every sequence of exact kernels clears it before its first quantisation."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "strata_b200", "csrc", "api.cu")


def test_range_flag_is_cleared_by_every_exact_call():
    text = open(SOURCE).read()
    calls = re.findall(r"(CK\(cudaMemsetAsync\(|launch_dsv4_quantize\(|launch_dsv4_gate_up\(|launch_dsv4_down\()([^;]*);", text)
    flag = r"\b(tiny|ctx->d_dsv4_tiny)\b"
    steps = [name for name, args in calls if re.search(flag, args)]
    one = ["CK(cudaMemsetAsync(", "launch_dsv4_quantize(", "launch_dsv4_gate_up(", "launch_dsv4_quantize(", "launch_dsv4_down("]
    assert steps == one * 2, steps       # routed experts, FP8 shared expert
