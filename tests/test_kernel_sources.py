"""Orderings that no run shows to be missing, read from the sources.

Shared memory of another CTA of a cluster may only be touched once that CTA is known to have started: every kernel that maps it
passes a cluster barrier first.  A kernel that reads before its dependency wait what an earlier pass wrote needs a plain
launch, which waits for everything, at the start of its own pass.  A named barrier has no limit, so no warp may skip it because one
of its limited waits has run out."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen-llm_b200", "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\([^;{]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            body = text[m.end():i]
            if "map_shared_rank" in body:
                yield os.path.basename(path), m.group(1), body


CASES = list(kernels())


def test_the_kernels_are_found():
    assert {"argmax_kernel", "gdn_mix_kernel", "tm_small_matmul_kernel"} <= {name for _, name, _ in CASES}


@pytest.mark.parametrize("file,name,body", CASES, ids=[c[1] for c in CASES])
def test_a_cluster_barrier_comes_before_remote_shared_memory(file, name, body):
    before = body[:body.index("map_shared_rank")]
    assert "cluster.sync()" in before or ("cluster.barrier_arrive()" in before and "cluster.barrier_wait()" in before), file
    # and one behind the last use, so that no CTA leaves while its shared memory is used
    assert "cluster.sync()" in body[body.rindex("map_shared_rank"):], file


def test_a_pass_starts_with_a_plain_launch():
    glue = open(os.path.join(CSRC, "glue.cu")).read()
    body = re.search(r"dfl_status launch_embed_block\(.*?\n}", glue, re.S).group(0)
    assert "embed_block_kernel<<<" in body and "launch_k(" not in body
    for path, fn in (("model.cu", "verify_core"), ("drafter.cu", "draft_core")):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
        core = text[re.search(r"dfl_status " + fn + r"\([^;{]*\{", text).end():]
        queued = re.findall(r"DFL_CHECK\((launch_\w+)\(", core)   # on the pass's own stream, in order
        assert queued[0] == "launch_embed_block", path


def _enclosing(text, at):
    """Headers of the blocks around a position, innermost first."""
    depth = 0
    for i in range(at, -1, -1):
        depth += {"}": 1, "{": -1}.get(text[i], 0)
        if depth < 0:
            depth = 0
            start = max(text.rfind(c, 0, i) for c in "{}\n")
            line = text.rfind("\n", 0, i) + 1
            yield text[min(start + 1, line):i]


def test_named_barriers_do_not_depend_on_a_limited_wait():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"named_sync\(1|bar\.sync 1,", text):
            seen += 1
            for header in _enclosing(text, m.start()):
                assert not re.search(r"\bok\b", header), (os.path.basename(path), header.strip())
    assert seen >= 8
