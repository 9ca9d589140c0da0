"""Rules of launches that can be looked at without a GPU: the host side of the kernel library, and its sources."""

import os
import re

import pytest


@pytest.fixture(scope="module")
def lib():
    from lily_b200.csrc import build, ops
    try:
        return ops.library()
    except build.BuildError as exc:
        pytest.skip(f"no kernel library here: {exc}")


def test_rows_over_clusters_take_whole_warps(lib):
    """Sums over the lanes of a warp name all 32 of them, so a block has whole warps, enough for its share of the row and no warp more."""
    taken = 0
    for width in range(4, 40000, 4):
        threads, pieces = lib.lily_row_cluster_threads(width), width // 32
        if width % 32 or not 32 <= pieces <= 1024:
            assert threads == 0
            continue
        taken += 1
        assert threads % 32 == 0 and pieces <= threads < pieces + 32 and threads <= 1024, width
    assert taken == 993


def test_no_block_writes_to_a_peer_that_may_not_have_started():
    """In every kernel that writes into the shared memory of other blocks of its cluster, a barrier that all of them have reached stands ahead of
    the first such write."""
    from lily_b200.csrc import build
    found = []
    for name in build.SOURCES:
        with open(os.path.join(build.HERE, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        # from one kernel's head to the next
        heads = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(heads, heads[1:]):
            body = text[a:b]
            write = re.search(r"map_shared_rank\([^;=]*=[^=]", body)
            if write is None:
                continue
            found.append(name)
            arrive, wait = body.find("cluster_arrive_started();"), body.find("cluster_wait_started();")
            assert 0 < arrive < wait < write.start(), (name, body[:200])
            assert body.count("cluster_arrive_started();") == body.count("cluster_wait_started();") == 1, name
    assert sorted(found) == ["attention_mma.cu", "combine.cu", "elementwise.cu", "elementwise.cu", "sublayer.cu"]


@pytest.mark.parametrize("shares,ff,lanes", [((None, None), True, 2), (("first", None), True, 2), (("first", "blend"), True, 0), (("blend", "blend"), False, 0),
                                             ((None, "blend", None), False, 2), (("first", "blend", None), True, 0)])
def test_mixers_that_meet_in_a_buffer_of_the_step_keep_their_order(shares, ff, lanes):
    """Attention mixers of one parallel block whose values are the first sharing layer's write and read one buffer of the step, so a captured
    step does not run them side by side."""
    import torch
    import kernel_refs
    from lily_b200.parts.attention import AttentionSpec
    from lily_b200.parts.base import BuildContext, build_part
    from lily_b200.parts.block import ParallelBlockSpec
    from lily_b200.parts.mlp import SwiGLUSpec
    from lily_b200.parts.norm import RMSNormSpec
    mixers = tuple((f"m{i}", AttentionSpec(32, 2, 1, 16, v_share=s), f"g{i}") for i, s in enumerate(shares))
    spec = ParallelBlockSpec("b", 32, mixers, SwiGLUSpec(32, 64) if ff else None, RMSNormSpec(32, 1e-6), 1e-6)
    ctx = BuildContext(torch.device("cpu"), torch.float32, kernel_refs)
    assert build_part("block", spec, "b", ctx).lanes == lanes


def test_the_recurrence_is_cut_for_the_kernels_that_take_it(lib):
    """Chunks from 33 tokens on are the tensor-core kernels': float32 and head sizes beyond theirs have the cut of before, and no scratch for
    portions that run whole."""
    import torch
    from lily_b200.csrc import ops
    for lens in ([100], [1, 33, 128], [20, 30]):
        for dtype, d in ((torch.float32, 64), (torch.bfloat16, 80), (torch.bfloat16, 128), (torch.bfloat16, 40)):
            plan = ops.wkv_plan(lens, "cpu", dtype, d)
            assert plan is None and ops.wkv_workspace_floats(plan, 4, d) == 0
    assert ops.wkv_plan([20, 30], "cpu") is None
    fine = ops.wkv_plan([1, 33, 128], "cpu", torch.bfloat16, 48)
    assert fine.items == 0 and fine.fine.items == 3 and fine.fine.shorts == 1
    for dtype, chunks in ((torch.float32, None), (torch.bfloat16, 1 + 2 + 4)):
        plan = ops.wkv_plan([1, 33, 128, 200], "cpu", dtype, 64)
        assert plan.items == 4 and plan.shorts == 3 and (plan.fine and plan.fine.items) == chunks
        assert plan.item_start.tolist() == [0, 64, 128, 192] and plan.item_len.tolist() == [64, 64, 64, 8] and plan.long_req.tolist() == [3]
        assert ops.wkv_workspace_floats(plan, 4, 64) == (chunks or 4) * 4 * (64 * 64 + 64)
