"""Waits of the kernels give up after a limit, in one warp and not in another; a barrier between such waits has no limit.  So
warps that share one must all reach it, and leave their loops on what it tells all of them."""
import os
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "memory_b200", "csrc")


def test_row_warps_of_the_token_mixture_leave_their_loop_at_the_barrier_only():
    text = open(os.path.join(CSRC, "token_mix_tc.cu")).read()
    kernel = text[text.index("token_mix_fwd_tc_kernel("):text.index("__global__ void slot_reduce_kernel")]
    rows = kernel[kernel.index("const int r = threadIdx.x;"):]          # what the row-owning warps run
    lines = [ln.strip() for ln in rows.splitlines()]
    meets = [i for i, ln in enumerate(lines) if "row_warps_agree(" in ln]
    exits = [i for i, ln in enumerate(lines) if re.search(r"\b(break|return|continue|goto)\b", ln)]
    assert len(meets) == 2 and "bar.sync" not in rows
    assert exits == meets[1:], "a way out that another warp need not take"


def test_a_step_whose_wait_ran_out_is_neither_read_nor_stored():
    """Backward of chapters with few pairs: the record of a step (where its results go) and its rows are written by another warp, so
    between the waits for them and the meeting of the warps everything that looks at them is under the outcome of the waits."""
    text = open(os.path.join(CSRC, "token_mix_rows.cuh")).read()
    kernel = text[text.index("token_mix_rows_bwd_kernel("):]
    loop = kernel[kernel.index("bool ok = mbar_wait_w(&full[buf]"):]
    meeting = "if (!warps_agree<1, 128>(halves > 0)) break;"
    assert loop.count("warps_agree") == loop.count(meeting) == 1
    way, behind = loop.split(meeting)
    assert "const int halves = !ok ? 0 : st.pairs > 16 ? 2 : 1;" in way
    start = way.index("if (warp < 2 * halves) {")
    depth = 0
    for end in range(way.index("{", start), len(way)):
        depth += {"{": 1, "}": -1}.get(way[end], 0)
        if depth == 0:
            break
    assert "p.d_w_heads[st.dw_at" in way[start:end]
    rest = re.sub(r"//[^\n]*", "", way[:start] + way[end + 1:]).replace("!ok ? 0 : st.pairs > 16 ? 2 : 1", "")
    assert not re.search(r"\bst\.|ldsm|stsm|\bp\.(?!status\b|dkv_ld\b)", rest), rest
    assert not re.search(r"\b(break|continue|goto)\b|\breturn;", way) and "break" not in behind[:behind.index("__syncthreads();")]


@pytest.mark.gpu
@pytest.mark.parametrize("late", [0, 1, 8, 6, 15])
def test_warps_agree_about_their_waits(late):
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    own, heard = ops.agree_probe(dev, late, 2000)
    assert own == [1 - ((late >> w) & 1) for w in range(4)] and heard == [int(late == 0)] * 4
    if late:
        with pytest.raises(RuntimeError, match="timed out"):
            L.check_device_status(dev)
    L.check_device_status(dev)


def test_no_warp_walks_a_whole_chapter_of_the_token_mixture_alone():
    """Forward of chapters with few pairs: routing may send every pair to a few of them, so an item is a tile of the index (at most 128
    pairs), as in the other kernel, and never a bucket."""
    text = open(os.path.join(CSRC, "token_mix_rows.cuh")).read()
    kernel = text[text.index("token_mix_rows_fwd_kernel("):text.index("// ---- backward")]
    assert "g.n = p.tile_cnt[tile];" in kernel and "bucket_off" not in kernel and "seek(" not in kernel
