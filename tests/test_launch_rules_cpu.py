"""Rules of launches that can be looked at without a GPU: the host side of the kernel library, and its sources."""

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
