"""Named and cluster barriers in the kernel sources: the aligned kinds (bar.*
always, barrier.* with .aligned) have to be executed by a warp as one, so each
comes straight after a __syncwarp(); the compiler's reconvergence after a
lane-dependent branch is no promise."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "ugsdr_gb300" / "csrc"
ALIGNED = re.compile(r'asm volatile\("[^"]*(?:(?<![\w.])bar\.(?:sync|arrive|red)|barrier[.\w:]*\.aligned)')


def test_aligned_barriers_follow_a_warp_convergence():
    found = 0
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        source = path.read_text()
        for m in ALIGNED.finditer(source):
            found += 1
            before = source[:m.start()].rstrip()
            assert before.endswith("__syncwarp();"), f"{path.name}: {source[m.start():m.end()]}"
    assert found >= 2  # the tracking bank's
