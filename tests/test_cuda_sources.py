"""Rules of the CUDA programming model that a run cannot show to be kept.

A missing barrier need not give a wrong result on any machine at hand, so
these read the kernels' source.
"""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "smili_b200", "csrc")


def _sources():
    out = {}
    for p in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(p) as f:
            out[os.path.basename(p)] = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
    return out


def _block(text, start):
    """The text from start to the brace that closes the first one opened after it."""
    i = text.index("{", start)
    depth = 0
    for k in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[i:k + 1]
    raise ValueError("unbalanced braces")


def _kernels():
    for name, text in _sources().items():
        for m in re.finditer(r"__global__[^{;]*", text):
            k = re.search(r"(\w+)\s*\((?:[^()]|\([^()]*\))*\)\s*$", m.group(0))
            if k:
                yield name, k.group(1), _block(text, m.end())


def test_kernels_are_found():
    names = {k for _, k, _ in _kernels()}
    assert {"smili_batch_kernel", "bias_grad_kernel", "conv3x3_tc_kernel", "uvsort_count"} <= names


def test_other_ctas_shared_memory_is_reached_after_a_cluster_barrier():
    """A CTA may not touch another's shared memory before that CTA is known to
    have started, nor leave while another may still touch its own."""
    barrier = re.compile(r"cluster\.sync\(\)|cluster\.barrier_wait\(\)")
    seen = 0
    for name, kernel, body in _kernels():
        remote = [m.start() for m in re.finditer(r"map_shared_rank|\bmapa\b", body)]
        if not remote:
            continue
        seen += 1
        waits = [m.start() for m in barrier.finditer(body)]
        assert waits and waits[0] < remote[0], f"{name}: {kernel}"
        assert waits[-1] > remote[-1], f"{name}: {kernel}"
    assert seen


def test_waits_before_warp_wide_instructions_answer_for_the_warp():
    """A role that a whole warp plays issues .aligned instructions (tcgen05.ld,
    elect, __syncwarp), so its bounded waits must end alike in every lane, also
    when one runs out: only a role of a single lane may wait by itself."""
    seen = 0
    for name, kernel, body in _kernels():
        if "tmem_ld16" not in body:
            continue
        seen += 1
        for m in reversed(list(re.finditer(r"lane == 0\)\s*(?=\{)", body))):
            block = _block(body, m.end())
            body = body[:m.end()] + body[m.end():].replace(block, "", 1)
        assert not re.search(r"\bmbar_wait\(", body), f"{name}: {kernel}"
    assert seen


def test_build_watches_every_included_file():
    """A library is rebuilt when any file its source includes has changed."""
    from smili_b200 import build
    for src, deps, hdrs in build.LIBS.values():
        found, todo = set(), [src]
        while todo:
            with open(os.path.join(CSRC, todo.pop())) as f:
                inc = {os.path.basename(i) for i in re.findall(r'#include\s+"([^"]+)"', f.read())}
            todo += [i for i in inc - found if os.path.exists(os.path.join(CSRC, i))]
            found |= inc
        assert found == set(deps) | set(hdrs)
