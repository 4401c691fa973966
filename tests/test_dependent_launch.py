"""A pass that is launched as a programmatic dependent is alive while the pass
before it still writes, so it may read by __ldg (ld.global.nc: memory that is
read-only for the life of the grid) only what no pass writes: the matrix and
its schedules in the kernels, the tiles' instances in the epilogues. Read off
the sources: a stale value would need an unlucky timing on the GPU."""

import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "vikalp_b200", "csrc")
SOURCES = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read())
           for p in glob.glob(os.path.join(CSRC, "*.cu*"))}


def _body(text, at):
    """The braces' content that opens at or after `at`."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced braces")


def _kernels():
    for name, text in SOURCES.items():
        for g in re.finditer(r"__global__[^{;]*?(\w+)\(", text):
            if g.group(1) in ("__launch_bounds__", "__cluster_dims__"):
                g = re.compile(r"\s*(?:__cluster_dims__\([^)]*\)\s*)?(\w+)\(").search(text, text.index(")", g.end()))
            end = text.index(")", g.end())
            if text[end + 1:].lstrip()[:1] == "{":  # a definition
                yield f"{name}: {g.group(1)}", _body(text, end)


def test_kernels_read_only_the_matrix_by_ldg():
    dependent = {k: b for k, b in _kernels() if "pdl_wait()" in b}
    names = {k.split(": ")[1] for k in dependent}
    assert {"tile_kernel_fast", "tile_kernel_sub", "tile_kernel_hyb", "tile_kernel_tma", "ref_control_kernel"} <= names
    for k, body in dependent.items():
        for arg in re.findall(r"__ldg\(\s*&?([\w.]+)", body):
            assert arg.startswith("M."), f"{k} reads {arg} by __ldg"
        assert not re.search(r"__restrict__\s+\w+\s*=\s*g\.p", body), k


def test_epilogues_read_only_the_instances_by_ldg():
    found = 0
    for name, text in SOURCES.items():
        for s in re.finditer(r"struct (\w+) : Epi(?:Base|Row)<", text):
            found += 1
            body = _body(text, s.end())
            assert "__restrict__" not in body, f"{name}: {s.group(1)}"
            for arg in re.findall(r"__ldg\(\s*&?([\w.>-]+)", body):
                assert arg == "tile_inst", f"{name}: {s.group(1)} reads {arg} by __ldg"
    assert found >= 20


def test_gathered_vectors_are_not_restrict():
    csr = SOURCES["vk_csr.cuh"]
    assert "__restrict__" not in _body(csr, csr.index("struct Gathers"))
