"""The ctypes mirror of the C ABI matches the header's struct layouts: a small C
program compiled against include/mapgraph_b200.h prints sizeof / offsetof of
every field of every public struct, and the ctypes structures must agree (CPU;
a mismatch would silently corrupt options and counters at the boundary)."""
import ctypes as C
import os
import subprocess

import pytest

from mirrorofmapgraph_b200 import _build
from mirrorofmapgraph_b200 import _lib as L

STRUCTS = {
    "mg_opts": L.MgOpts,
    "mg_stats": L.MgStats,
    "mg_pr_opts": L.MgPrOpts,
    "mg_part_level": L.MgPartLevel,
    "mg_level_record": L.MgLevelRecord,
    "mg_host_csr": L.MgHostCsr,
    "mg_tuning": L.MgTuning,
}


def _c_layout(tmp_path):
    lines = ['#include <stddef.h>', '#include <stdio.h>', '#include "mapgraph_b200.h"',
             '#include "mapgraph_b200_io.h"', "int main(void) {"]
    for cname, cls in STRUCTS.items():
        lines.append(f'  printf("{cname} size %zu\\n", sizeof({cname}));')
        for fname, _ in cls._fields_:
            lines.append(f'  printf("{cname} {fname} %zu\\n", offsetof({cname}, {fname}));')
    lines += ["  return 0;", "}"]
    src = tmp_path / "layout.c"
    src.write_text("\n".join(lines) + "\n")
    exe = tmp_path / "layout"
    r = subprocess.run(["gcc", "-std=c11", "-I" + _build.INCLUDE, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail("layout probe did not compile:\n" + r.stderr)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    got = {}
    for line in out.splitlines():
        parts = line.split()
        got[tuple(parts[:-1])] = int(parts[-1])
    return got


def test_ctypes_structs_match_the_header(tmp_path):
    got = _c_layout(tmp_path)
    for cname, cls in STRUCTS.items():
        assert got[(cname, "size")] == C.sizeof(cls), cname
        for fname, _ in cls._fields_:
            assert got[(cname, fname)] == getattr(cls, fname).offset, (cname, fname)


def test_batched_sssp_row_offsets_past_32_bits(tmp_path):
    """Offsets into the interleaved distance rows (mss_row), and that the kernels use nothing else: a
    vertex from 2^27 on lies past 2^32 distances, on a graph too large for a test."""
    rows = [0, 1, 2**26 - 1, 2**26, 2**27 - 1, 2**27, 140_000_000, 2**31 - 1, 2**33]
    src = tmp_path / "rows.cu"
    src.write_text('#include "mg_internal.h"\nint main() {\n' +
                   "".join(f'  printf("%lld\\n", (long long)mss_row({r}ll));\n' for r in rows) + "}\n")
    exe = tmp_path / "rows"
    r = subprocess.run([_build.NVCC] + _build.NVCC_FLAGS + [str(src), "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail("row offset probe did not compile:\n" + r.stderr)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert [int(x) for x in out.split()] == [32 * r for r in rows]
    with open(os.path.join(_build.CSRC, "sssp.cu")) as f:
        text = f.read()
    assert text.count("<< 5") == text.count("(tile % vtiles) << 5")  # a tile's first vertex
