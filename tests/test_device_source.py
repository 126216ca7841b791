"""Rules of the device code that no run can show to be kept: what breaks them is
undefined on the GPU (it works until a compiler orders the lanes differently), so the
sources are checked instead."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "inverse-solver-gpu_b200", "csrc", "*.cu*")))


def _code(path):
    """The file without comments, its lines where they were."""
    with open(path) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)


def test_aligned_instructions_converge_the_warp_first():
    """An .aligned instruction (bar.sync is one) run by part of a warp is undefined: every
    function that issues one calls __syncwarp() before it."""
    found, bad = 0, []
    for path in SOURCES:
        code = _code(path)
        for m in re.finditer(r'"[^"\n]*(?:\.aligned|bar\.sync)[^"\n]*"', code):
            found += 1
            start = max(code.rfind("__device__", 0, m.start()), code.rfind("__global__", 0, m.start()))
            if "__syncwarp()" not in code[start:m.start()]:
                bad.append(f"{os.path.basename(path)}:{code.count(chr(10), 0, m.start()) + 1}")
    assert found >= 8
    assert not bad, bad
