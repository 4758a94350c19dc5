"""Properties of the kernel sources that no call can show: paths that are taken after a failed launch only."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "llm_from_scratch_b200" / "csrc"


def test_a_failed_launch_leaves_no_error_behind():
    """Every launch with attributes goes through the helper that clears the runtime's last error."""
    calls = [(p.name, m.start()) for p in CSRC.glob("*.cu*") for m in re.finditer(r"cudaLaunchKernelEx\(", p.read_text())]
    through = [(p.name, m.start(1)) for p in CSRC.glob("*.cu*")
               for m in re.finditer(r"return launch_result\((cudaLaunchKernelEx\()", p.read_text())]
    assert calls and calls == through


def test_no_cta_leaves_while_its_bulk_copies_may_be_on_their_way():
    """A wait that ran out ends the delta scans behind a barrier that all threads leave with one answer and a bounded wait for
    the copies; no thread decides by a flag that another may set behind the barrier."""
    text = (CSRC / "delta_chunk.cu").read_text()
    scan, split = (text[text.index(f"{k}(const ChunkArgs args"):] for k in ("delta_scan_kernel", "delta_split_kernel"))
    for body in (scan[:scan.index("struct SplitLayout")], split[:split.index("EncodeFn")]):
        assert "all_landed(" in body and not re.search(r"if \(s_abort\)|return s_abort", body)
    helper = text[text.index("bool all_landed("):]
    helper = helper[:helper.index("\n}\n")]
    at = [helper.index(x) for x in ("__syncthreads_or(!here)", "mbar_wait(bar", "__syncthreads();", "return false")]
    assert at == sorted(at)
