"""Kernels start before the one ahead of them on the stream is complete (csrc/launch.cuh), so every kernel waits for it
itself: first thing, or after a set-up of barriers and tensor memory that touches no global memory."""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "see_ai_b200" / "csrc"
SETUP = re.compile(r"MbarInit|TmemAlloc|tcgen05\.(alloc|relinquish)")


def _bodies(text):
    """(name, parameters, body) of every __global__ function of a source."""
    for m in re.finditer(r"^\s*(?:template <[^;{]*>\s*)?__global__", text, re.M):
        at = text.index("(", m.end())
        while True:
            name = re.search(r"(\w+)\s*$", text[m.end():at]).group(1)
            depth, end = 0, at
            while True:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                if depth == 0:
                    break
                end += 1
            if name != "__launch_bounds__":
                break
            at = text.index("(", end)
        begin = text.index("{", end)
        depth, close = 0, begin
        while True:
            depth += {"{": 1, "}": -1}.get(text[close], 0)
            if depth == 0:
                break
            close += 1
        yield name, text[at + 1:end], text[begin + 1:close]


def test_every_kernel_awaits_the_one_before_it():
    kernels = 0
    for path in sorted(CSRC.glob("k_*.cu")):
        text = path.read_text()
        if path.name == "k_no_alloc.cu":   # plain launches on the caller's stream
            assert "Next(" not in text
            continue
        assert "<<<" not in text.replace("kernel<<<grid", ""), path.name
        for name, params, body in _bodies(text):
            kernels += 1
            assert body.count("AwaitPrevious();") == 1, (path.name, name)
            before = body[:body.index("AwaitPrevious();")]
            if not before.strip():
                continue
            assert SETUP.search(before), (path.name, name)
            # What runs earlier reads no pointer it was given (tensor maps and scalars are the launch's own).
            for p in re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*(?:,|$)", params):
                assert not re.search(rf"\b{p}\s*\[|\*{p}\b|__ldg\(.*\b{p}\b", before), (path.name, name, p)
            assert not re.search(r"__ldg|TmaLoad|LoadRows|\bld\.global|cp\.async\.bulk", before), (path.name, name)
    assert kernels > 60
