"""Waits that the kernels must not miss, read from their sources: what they guard against (an arrival in shared memory that belongs to
another CTA by then, a warp whose lanes part) shows in no result, and provoking it would hang or corrupt a GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gemm_int8_b200", "csrc")


def _kernels():
    """(name, body) of every kernel that issues tensor-core work, comments removed."""
    found = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cuh"):
            continue
        with open(os.path.join(CSRC, f)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__[^;{]*?\n(\w+)\(const __grid_constant__", text):
            body = text[m.end():text.index("\n}\n", m.end())]
            if "umma_commit" in body:
                found.append(pytest.param(body, id=m.group(1)))
    return found


def test_all_kernels_are_seen():
    names = {p.id for p in _kernels()}
    assert names == {"dense_gemm_kernel", "dense_splitk_kernel", "smallm_gemm_kernel", "smallm_cluster_kernel", "blockwise_gemm_kernel",
                     "blockwise_smallm_kernel"}


@pytest.mark.parametrize("body", _kernels())
def test_last_commits_are_awaited(body):
    """The barrier that the issuer's commits hand a stage back on is waited for to the last of them, by the producer of each CTA."""
    ring = "bar_done" if re.search(r"\bbar_done\[", body) else "bar_empty"
    assert re.search(r"umma_commit\(&%s\[|umma_commit_pair\(map_to_cta\((smem_u32\(&%s\[|done_0)" % (ring, ring), body)
    drains = re.findall(r"drain_stages<STAGES(?:, DONE_RINGS)?>\(([^;]*)\);", body)
    assert len(drains) == 1 and re.search(r"bar_full, %s(\[0\])?, " % ring, drains[0])


def test_staging_blocks_alternate_from_store_to_store():
    """tma_store_wait_read<1> leaves the warp's latest store unread: the block staged next must be the other one, also when the latest store was
    the last of an odd number in its tile.  So the dense kernel picks it by a count of its stores and not by the column."""
    body = {p.id: p.values[0] for p in _kernels()}["dense_gemm_kernel"]
    assert "tma_store_wait_read<1>" in body
    pick = re.search(r"stg = store_stage \+ ([^;]*);", body).group(1)
    assert "staged++" in pick and not re.search(r"\bc\b", pick)
    assert "staged = 0" not in body.split("for (int tile = first_tile; tile < num_tiles && ok; tile += tile_step, ++local_tile) {")[-1]


@pytest.mark.parametrize("body", _kernels())
def test_lanes_of_a_warp_decide_together(body):
    """Full-mask instructions stand behind every bounded wait, so whether it has failed is a vote (only the roles of a single thread do without)."""
    waits = 0
    for m in re.finditer(r"\bwait_or_abort(?:_addr)?\(", body):
        start = max(body.rfind(c, 0, m.start()) for c in ";{}")
        end = m.start() + re.search(r"[;{]", body[m.start():]).start()
        statement = body[start + 1:end]
        if "const bool ready =" in statement:
            statement = body[start + 1:body.index(";", end + 1)]
            assert "warp_agrees(ready," in statement
        if "warp_agrees(" not in statement:
            role = body[:start].rfind("if (lane == 0")
            assert role > body[:start].rfind("} else if (warp == ") and "elect_one" not in body[role:start], statement
        waits += 1
    assert waits >= 3


def test_remote_stores_follow_a_barrier_of_the_cluster():
    """A peer's shared memory may be written only once its CTA has started: some cluster barrier lies before the first remote store."""
    for p in _kernels():
        m = re.search(r"\bst_dsmem_\w+\(", p.values[0])
        if m:
            assert re.search(r"\bcluster_(sync_all|wait)\(\)", p.values[0][:m.start()]), p.id
