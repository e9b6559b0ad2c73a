"""Bounded waits of the kernels: where the lanes of a warp meet (elect.sync, __syncwarp, votes, shuffles), a wait that runs out must take the
whole warp along, or the lanes that were served wait for the others without a limit.  Read from the sources, since no test may make a
kernel stand still: in functions where lanes meet nothing is decided by a wait's result before the warp has voted on it.  (What waits for
copies in flight once all is lost does not use it.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tile_fusion_b200", "csrc")
WAIT = re.compile(r"\b(?:mbar_try|mbar_wait|wait_or_abort|pair_wait(?:<\w+>)?)\(")
MEET = re.compile(r"__syncwarp|elect_one\(|elect_lane\(|__all_sync|__shfl|\.sync\.")


def _functions(text):
    """Top-level definitions: from a line that opens one in the first column to the closing brace there."""
    return re.findall(r"^(?:template|__global__|__device__|static|bool|int)[^\n;]*\n(?:(?!\}).*\n)*\}", text, re.M)


def _offences(text):
    out = set()
    for f in _functions(text):
        body = f[f.index("{"):] if "{" in f else ""
        if not MEET.search(body):
            continue
        open_result = False  # `ok` holds a result that has not been voted on
        for line in 2 * body.splitlines():  # (twice: a loop may come round with one)
            code = line.split("//")[0]
            if WAIT.search(code) and "__all_sync(" not in code:
                if re.match(r"\s*(?:for \(.*\)\s*)?(?:%s)" % WAIT.pattern, code) or re.search(r"for \(.*!mbar_wait\(.*\+\+k\) \{\}", code):
                    continue  # not used
                if re.match(r"\s*(?:if \(.*\) )?ok &?= ", code):
                    open_result = True
                else:
                    out.add(line.strip())
            elif open_result and re.search(r"\bok\b", code):
                if re.search(r"__all_sync\(\w+, ok\)", code):
                    open_result = False
                elif re.search(r"\b(?:if|for|while|return)\b|\?", code):
                    out.add(line.strip())
    return sorted(out)


@pytest.mark.parametrize("source", ["band_march.cu", "lattice_march.cu", "row_gemm.cu", "spmm_gemm.cu", "tile_pipeline.cu"])
def test_a_warp_leaves_as_one(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    assert len(_functions(text)) > 3 and WAIT.search(text)
    assert _offences(text) == []


def test_what_is_looked_for():
    kernel = "__global__ void k(int *p) {\n  bool ok = true;\n  %s\n  if (ok) *p = 1;\n  __syncwarp();\n}\n"
    assert _offences(kernel % "ok = mbar_wait(bar, 0, limit);")
    assert _offences(kernel % "ok &= mbar_wait(bar, 0, limit);")
    assert _offences(kernel % "if (!wait_or_abort(bar, 0, limit, abort)) return;")
    assert not _offences(kernel % "ok = __all_sync(kFull, mbar_wait(bar, 0, limit));")
    assert not _offences(kernel % "ok = mbar_wait(bar, 0, limit);\n  if (!(ok = __all_sync(kFull, ok))) return;")
    assert not _offences(kernel % "mbar_wait(bar, 0, limit);")
    assert not _offences((kernel % "ok = mbar_wait(bar, 0, limit);").replace("__syncwarp();", "__syncthreads();"))
