"""CPU checks of the device sources for mistakes that could hang a GPU and that
no run shows reliably."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "c-saw_b200", "csrc", "*.cu*")))


def test_inline_barriers_need_no_convergence():
    """bar.sync, bar.red, bar.arrive and barrier.*.aligned are defined only when
    all threads of a warp reach them together.  In inline PTX nothing tells the
    compiler to bring the warp together first, so the sources use the
    barrier.* forms without .aligned there."""
    assert SOURCES
    found = 0
    for path in SOURCES:
        for asm in re.findall(r'asm\s+(?:volatile\s*)?\(\s*((?:"[^"]*"\s*)+)', open(path).read()):
            for op in re.findall(r"\bbar(?:rier)?\.[a-z0-9_.]+", asm):
                found += 1
                assert op.startswith("barrier.") and ".aligned" not in op, (os.path.basename(path), op)
    assert found
