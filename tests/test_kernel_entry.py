"""Launches that overlap (programmatic dependent launch): completion is passed on from kernel to kernel, so that every kernel of the stream has to wait for the one before it in
every thread (pdl_enter), before it returns and before it writes.  CPU only: the sources are read."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crabml_b200", "csrc")


def body(text, at):
    """the braces that open at text[at]"""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError("unbalanced braces")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+", text):
            after = re.sub(r"(__launch_bounds__|__cluster_dims__)\s*\((?:[^()]|\([^()]*\))*\)\s*", lambda g: " " * len(g.group()), text[m.end():m.end() + 4000])
            name = re.match(r"\s*(\w+)\s*\(", after)
            if name:
                yield os.path.basename(path), name.group(1), body(text, text.index("{", m.end() + name.end()))


def test_no_kernel_returns_before_it_has_waited():
    seen = 0
    for path, name, code in kernels():
        if "pdl_enter();" not in code:
            continue
        seen += 1
        before = code[:code.index("pdl_enter();")]
        while (m := re.search(r"\[[&=]?\]\s*\([^()]*\)\s*(?:->\s*\w+\s*)?\{", before)):       # what a lambda returns stays in it
            inner = body(before, m.end() - 1)
            before = before[:m.start()] + before[m.end() - 1 + len(inner):]
        assert not re.search(r"\breturn\b", before), (path, name)
    assert seen > 60


def test_every_kernel_of_an_overlapping_launch_waits():
    waits = {name for _, name, code in kernels() if "pdl_enter();" in code}
    every = {name for _, name, _ in kernels()}
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"cc_launch_(?:pdl|alone|when)\s*\((?:[^,]*,)?\s*dev\s*,\s*([^,;]*)", text):
            for name in set(re.findall(r"\b(\w+_kernel)\b", m.group(1))) & every:
                assert name in waits, (os.path.basename(path), name)
