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
