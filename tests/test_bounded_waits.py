"""How the roles of the tensor-core expert kernel leave after a wait that ran out, read from the source: threads that meet
at a barrier or in a warp-wide instruction must take the decision to leave together (a time-out itself is not provoked)."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "strata_b200", "csrc", "prefill.cu")


def role(title):
    """Source of one role of prefill_ffn_kernel: from its title line to the next one's (or the tile list)."""
    text = open(SOURCE).read()
    parts = re.split(r"// -{20,} ", text[text.index("__global__ void __launch_bounds__(kThreads, 1)"):])
    found = [p for p in parts if p.startswith(title)]
    assert len(found) == 1, title
    return found[0].split("tc_fence_before();\n    __syncthreads();")[0]


def test_epilogue_warps_share_one_verdict():
    body = role("epilogue")
    assert "*abort_flag)" not in body           # nobody decides on a flag that another role may raise meanwhile
    assert body.count("mbar_wait(") == 1 and re.search(r"if \(epilogue_vote\(ew == 0u && !mbar_wait\(", body)
    assert re.search(r"epilogue_vote\(.*\)\) \{ ok = false; break; \}", body)


def test_lanes_of_decoders_and_issuers_leave_together():
    body = role("weight decoders")
    assert body.count("mbar_wait_warp(") == 2 and "mbar_wait(" not in body
    body = role("MMA issuers")
    assert len(re.findall(r"if \(!all\((got|mbar_wait\(.*\))\)\) \{ ok = false; break; \}", body)) == 2
