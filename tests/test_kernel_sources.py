"""Orderings that no run shows to be missing, read from the sources.

Shared memory of another CTA of a cluster may only be touched once that CTA is known to have started: every kernel that maps it
passes a cluster barrier first.  A kernel that reads before its dependency wait what an earlier pass wrote needs a plain
launch, which waits for everything, at the start of its own pass.  A kernel that starts without a dependency wait acquires what the
kernel before published behind its own, and waits at its end.  A named barrier has no limit, so no warp may skip it because one
of its limited waits has run out."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen-llm_b200", "csrc")


def all_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\([^;{]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield os.path.basename(path), m.group(1), text[m.end():i]


CASES = [k for k in all_kernels() if "map_shared_rank" in k[2]]


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


def test_launches_without_a_dependency_wait_acquire_a_mark():
    # launch_dependents orders no memory: what a grid two launches back wrote is read behind an acquire of the word that the grid between
    # released behind its own wait
    readers = {name: body for _, name, body in all_kernels() if "late_acquire(" in body}
    assert set(readers) == {"gemm_ts_kernel", "ab_proj_kernel"}
    gemm = readers["gemm_ts_kernel"]
    assert "if (p.late_mode == LATE_BEHIND) late_acquire(" in gemm
    assert "if (p.late_mode == LATE_BEHIND) pdl_wait();" in gemm[gemm.index("tmem_free("):]   # waits at its end
    assert gemm.count("pdl_launch_dependents()") == 2 and "if (p.late_mode != LATE_FIRST) pdl_launch_dependents();" in gemm
    trigger = gemm[gemm.index("auto trigger"):]
    assert trigger.index("pdl_wait()") < trigger.index("pdl_launch_dependents()")
    publish = gemm.index("late_publish(")
    assert re.search(r"trigger\(\);\s*if \(p\.late_mode == LATE_FIRST && blockIdx\.x == gridDim\.x - 1 && lane == 0\) $", gemm[:publish])   # behind the wait in trigger
    copies = gemm.index("bulk_g2s(acts_res")
    assert gemm.rindex('"fence.proxy.async.global;"', 0, copies) > gemm.rindex("wait_inputs();", 0, copies)
    ab = readers["ab_proj_kernel"]
    assert ab.index("late_acquire(") < ab.index("__ldcg(") and "if (late.word) pdl_wait();" in ab[ab.index("ab_part[("):]
    # who is launched so: one GEMM with the late trigger, then only such kernels, then an ordinary one
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "model.cu")).read())
    spans = [text[m.start():] for m in re.finditer(r"const bool late =", text)]
    assert len(spans) == 2 and text.count("trigger_late = ") == 2 and text.count("next_mark()") == 2
    queued = [re.findall(r"DFL_CHECK\((launch_\w+)\(([^;]*)\);", s) for s in spans]
    assert [q[0] for q in queued[0][:3]] == ["launch_gemm_fewrow", "launch_ab_proj", "launch_gdn_mix"]
    assert "ep.trigger_late = i == 0 && late;" in spans[0] and "ep.behind_late = i > 0 && late;" in spans[0] and "mark" in queued[0][1][1]
    assert [q[0] for q in queued[1][:2]] == ["launch_group", "launch_group"] and "ep_down, s->err" in queued[1][0][1] and "ep_down_exps, s->err" in queued[1][1][1]
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        if os.path.basename(path) != "model.cu":
            assert not re.search(r"\.(trigger|behind)_late = (?!ep\.)", open(path).read()), path


def test_kernels_of_the_chain_wait_before_they_read():
    launched = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        launched |= set(re.findall(r"\blaunch_k\(\s*(\w+_kernel)\b", re.sub(r"//[^\n]*", "", open(path).read())))
    waits = {name for _, name, body in all_kernels() if re.search(r"pdl_prologue\(\)|pdl_wait\(\)", body)}
    assert len(launched) > 20 and launched <= waits, launched - waits


def test_the_side_stream_s_kernels_do_not_run_ahead_of_their_wait():
    # they start behind an event, a full dependency: there is nothing to hide a second run of the code behind
    model = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "model.cu")).read())
    assert set(re.findall(r"(launch_\w+)\(side,", model)) == {"launch_small_matmul", "launch_moe_route"}
    bodies = {name: body for _, name, body in all_kernels()}
    for name in ("small_matmul_kernel", "moe_route_kernel"):
        assert "pdl_prologue();" in bodies[name] and not re.search(r"\bpass\b", bodies[name]), name


def test_both_routing_kernels_have_both_register_widths():
    moe = open(os.path.join(CSRC, "moe.cu")).read()
    for kernel in ("moe_route_kernel", "moe_route_lists_kernel"):
        assert re.search(r"n_expert <= ROUTE_NARROW \? " + kernel + r"<ROUTE_NARROW / 32> : " + kernel + r"<MOE_MAX_EXPERTS / 32>", moe), kernel


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
