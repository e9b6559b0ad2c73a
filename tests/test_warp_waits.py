"""Bounded waits of the kernels: where the lanes of a warp meet (elect.sync, __syncwarp, votes, shuffles), a wait that runs out must take the
whole warp along, or the lanes that were served wait for the others without a limit.  Read from the sources, since no test may make a
kernel stand still: in such functions a wait's result is voted on, or not used (what waits for copies in flight once all is lost)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tile_fusion_b200", "csrc")
WAIT = re.compile(r"\b(?:mbar_wait|wait_or_abort|pair_wait(?:<\w+>)?)\(")
MEET = re.compile(r"__syncwarp|elect_one\(|elect_lane\(|__all_sync|__shfl|\.sync\.")


def _functions(text):
    """Top-level definitions: from a line that opens one in the first column to the closing brace there."""
    return re.findall(r"^(?:template|__global__|__device__|static|bool|int)[^\n;]*\n(?:(?!\}).*\n)*\}", text, re.M)


def _offences(text):
    out = []
    for f in _functions(text):
        body = f[f.index("{"):] if "{" in f else ""
        if not MEET.search(body):
            continue
        lines = body.splitlines()
        for i, line in enumerate(lines):
            code = line.split("//")[0]
            if not WAIT.search(code) or "__all_sync(" in code:
                continue
            unused = re.match(r"\s*(?:for \(.*\)\s*)?(?:%s)" % WAIT.pattern, code) or re.search(r"for \(.*!mbar_wait\(.*\+\+k\) \{\}", code)
            soon = any("__all_sync(kFull, ok)" in x for x in lines[i + 1:i + 3])  # (two waits, one vote)
            if not unused and not soon:
                out.append(line.strip())
    return out


@pytest.mark.parametrize("source", ["band_march.cu", "row_gemm.cu", "spmm_gemm.cu", "tile_pipeline.cu"])
def test_a_warp_leaves_as_one(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    assert len(_functions(text)) > 3 and WAIT.search(text)
    assert _offences(text) == []


def test_what_is_looked_for():
    kernel = "__global__ void k(int *p) {\n  bool ok = true;\n  %s\n  __syncwarp();\n}\n"
    assert _offences(kernel % "ok = mbar_wait(bar, 0, limit);")
    assert _offences(kernel % "if (!wait_or_abort(bar, 0, limit, abort)) return;")
    assert not _offences(kernel % "ok = __all_sync(kFull, mbar_wait(bar, 0, limit));")
    assert not _offences(kernel % "mbar_wait(bar, 0, limit);")
    assert not _offences((kernel % "ok = mbar_wait(bar, 0, limit);").replace("__syncwarp();", "__syncthreads();"))
