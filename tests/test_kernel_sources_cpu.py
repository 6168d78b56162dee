"""Properties of the kernels' sources that no run can show without hanging a GPU."""
import re

from pisceslx_b200.ops import build


def test_blocks_agree_on_whether_a_wait_ran_out():
    """A thread's own read of the status word decides nothing but the end of its own wait; whatever a barrier follows asks
    the whole block (``block_gave_up``)."""
    for path in sorted(build.CSRC.iterdir()):
        code = re.sub(r"//[^\n]*", "", path.read_text()) if path.is_file() else ""
        reads = re.findall(r"volatile uint32_t\s*\*\s*>\s*\(\s*(?:p\.)?status\s*\)", code)
        assert len(reads) == (1 if path.name == "sm100.cuh" else 0), path.name
        for line in re.findall(r"[^\n]*\bgave_up\([^\n]*", code):
            assert "return false" in line or "bool gave_up" in line or "__syncthreads_or" in line, (path.name, line)
