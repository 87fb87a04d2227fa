"""What the kernels' sources must keep to, read as text."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmx_b200", "csrc")


def test_whole_warps_wait_with_a_vote():
    """A wait on an mbarrier gives up after a limit.  Where a whole warp waits and goes on to warp-wide instructions (tensor-memory
    loads, shuffles, votes), its lanes must not give up one by one: consumers', softmax and epilogue warps wait by
    `mbar_wait_warp` (or, latent_prompt_tc.cu, by a vote over the four warps).  A wait names its kind by its error code."""
    by_warps = re.compile(r"tc::mbar_wait\((?:[^()]|\([^()]*\))*\b(ERR_\w*(?:CONSUMER|SOFTMAX|EPILOGUE|ROWS))\b")
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        for number, line in enumerate(open(path, encoding="utf-8"), 1):
            m = by_warps.search(line)
            if m:
                found.append((os.path.basename(path), number, m.group(1)))
    assert not found, found


def test_no_call_lowers_a_kernels_limit_of_shared_memory():
    """The limit belongs to the function: a call that sets it to its own size can lower it under another thread's launch.  It is set to
    a constant (or, `allow_all_smem`, to all that there is)."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = open(path, encoding="utf-8").read()
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*?)\)\s*(?:;|!=|==|\)|\|\|)", text):
            value = m.group(1).strip()
            if not re.fullmatch(r"(?:\w+(?:<[^>]*>)?::)?[A-Z][A-Z_0-9]*", value) and os.path.basename(path) != "common.cuh":
                found.append((os.path.basename(path), text.count("\n", 0, m.start()) + 1, value))
    assert not found, found
