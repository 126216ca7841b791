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


def _role(code, at):
    """The text of the innermost block around `at` that an `if (warp == ...` opens."""
    depth, start = 0, at
    while start > 0:
        start -= 1
        if code[start] == "}":
            depth += 1
        elif code[start] == "{":
            depth -= 1
            if depth < 0:
                head = code[max(code.rfind(c, 0, start) for c in ";{}") + 1:start]
                if re.search(r"if\s*\(warp == ", head):
                    break
                depth = 0
    depth, end = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(code[end], 0)
        end += 1
        if depth == 0:
            return code[start:end]


def test_mma_warps_branch_on_votes():
    """elect.sync and votes take the whole warp.  A bounded wait can expire in some lanes and
    not in others, so in a warp that elects a lane no branch or loop depends on a wait's own
    result, only on a vote over it."""
    roles, bad = set(), []
    for path in SOURCES:
        code = _code(path)
        for m in re.finditer(r"if \(elect_one\(\)\)", code):
            role = _role(code, m.start())
            if role in roles:
                continue
            roles.add(role)
            own = r"\b(?:%s)\b" % "|".join(re.findall(r"(\w+) = mbar_wait(?:_or)?\(", role) + ["mbar_wait_or", "mbar_wait"])
            voted = re.sub(r"__all_sync\(0xffffffffu, \w+\)", "vote", role)
            bad += [(os.path.basename(path), head) for head in re.findall(r"(?:if|while) \([^\n]*|for \([^\n]*", voted)
                    if re.search(own, head)]
    assert len(roles) == 6
    assert not bad, bad


def test_waits_for_the_kernel_before_reach_every_address():
    """Read-only loads may be moved ahead of griddepcontrol.wait unless their address depends
    on it: grid_wait()'s zero goes into the block index, which is not read again without it,
    or into every pointer to what an earlier kernel may have written."""
    kernels, bad = 0, []
    for path in SOURCES:
        code = _code(path)
        starts = [m.start() for m in re.finditer(r"__global__", code)] + [len(code)]
        for a, b in zip(starts, starts[1:]):
            body = code[a:b]
            if "grid_wait()" not in body:
                continue
            kernels += 1
            index = re.search(r"(blockIdx\.[xyz]) \+ grid_wait\(\)", body)
            ok = index and body.count(index.group(1)) == 1
            if not index and re.search(r"\bz = grid_wait\(\);", body):
                args = re.findall(r"const (?:float2|int) \*__restrict__ (\w+)", body[:body.index("{")])
                tables = {"nearW", "basisT"}
                ok = len(args) > 2 and all(re.search(r"\b%s \+= z\b" % p, body) for p in args if p not in tables)
            if not ok:
                bad.append((os.path.basename(path), body[:body.index("{")][-60:]))
    assert kernels >= 20
    assert not bad, bad
