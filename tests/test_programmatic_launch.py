"""Kernels brought in beside their predecessor (launch_after) read what it wrote by load_written only: read-only loads
(__ldg, const __restrict__ parameters) promise memory that nothing writes while the kernel runs.  A wrong read of this
kind depends on timing, so the sources are read instead."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "miniisosurface_gb300" / "csrc"

# per kernel: the buffers that the kernel right before it in the stream writes
WRITTEN_BEFORE = {
    "k_scan_small": ["rowcnt", "mccnt"],                  # by the count
    "k_scan_partial": ["rowcnt", "mccnt"],
    "k_scan_final": ["part"],                             # by k_scan_partial
    "k_gen_cells": ["row4", "totals"],                    # by the scan, with rs.starts
    "k_vertices": ["points"],                             # by the generate kernel: its records
    "k_mc_remap": [],                                     # after the vertex kernel, which writes nothing it reads
}
# the same buffers where the kernels' bodies read them: row starts and first ids through walking pointers
BODIES = {
    "count_kernels.cu": ("__device__ __forceinline__ void load_counts", "// The Flying Edges scans of a list",
                         [r"rowcnt \+ b \+ q\b(?!\))", r"rowcnt \+ r\b", r"rowcnt\[", r"mccnt", r"part\b"]),
    "gen_cells.cuh": ("__device__ __forceinline__ void gen_cells_item", "// The warp's next work item",
                      [r"qp\b", r"sp\b"]),
}


def source(name):
    return (CSRC / name).read_text()


def test_every_programmatic_kernel_is_listed():
    text = "\n".join(p.read_text() for p in sorted(CSRC.glob("*.cu*")))
    named = set(re.findall(r"launch_after\(\s*(k_\w+)", text))
    if re.search(r"launch_after\(kern\b", text):  # launch_gen_cells picks an instantiation
        named.add("k_gen_cells")
    assert named == set(WRITTEN_BEFORE)


def test_parameters_are_not_read_only():
    text = "\n".join(p.read_text() for p in sorted(CSRC.glob("*.cu*")))
    for kernel, buffers in WRITTEN_BEFORE.items():
        head = re.search(r"__global__[^;{]*?\b%s\(([^{;]*)\)\s*\{" % kernel, text, re.S)
        assert head, kernel
        for b in buffers:
            p = re.search(r"([^,(]*)\b%s\s*(?:,|$)" % b, head.group(1))
            assert p, (kernel, b)
            assert not ("const" in p.group(1) and "__restrict__" in p.group(1)), (kernel, p.group(0).strip())


def test_bodies_read_them_coherently():
    for name, (begin, end, reads) in BODIES.items():
        text = source(name)
        body = text[text.index(begin):text.index(end)]
        for r in reads:
            assert not re.search(r"__ldg\(\s*&?\s*(?:%s)" % r, body), (name, r)
