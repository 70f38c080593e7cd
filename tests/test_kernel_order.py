"""Ordering rules of the kernels that no run can show (no GPU).

A missing warp barrier or fence lets a lane run ahead once in many runs, if at
all, so these rules are read off the sources: each test finds the place that
has to be ordered and looks for what orders it.
"""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "shearwave_b200" / "csrc"


def _source(name):
    """A source file without comments, white space collapsed."""
    text = (CSRC / name).read_text()
    return re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", text))


def _body(text, head):
    """The braces that follow the first match of ``head``."""
    start = text.index("{", re.search(head, text).end())
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError(head)


def test_neighbours_progress_is_ordered_before_the_copies():
    # 27 lanes acquire a neighbour's word each, one lane issues the copies;
    # a vote between them orders no memory
    body = _body(_source("sw_step_tb.cu"), r"bool tb_wait_around\([^{]*")
    done = body.index("v >= need")
    assert "__syncwarp()" in body[done:body.index("return true", done)]


@pytest.mark.parametrize("name", ["sw_project.cu", "sw_step_tb.cu", "sw_step_tma.cu"])
def test_a_warp_leaves_a_stage_together(name):
    # lane 0 frees a ring stage for its warp: not while another lane still
    # reads the stage, its slot or its barrier's phase
    text = _source(name)
    frees = [m.start() for m in re.finditer(r"mbar_arrive\(&[\w.>-]*empty", text)]
    assert frees
    for at in frees:
        guard = text.rindex("if (lane == 0)", 0, at)
        assert text[:guard].rstrip().endswith("__syncwarp();"), text[guard - 120:at + 40]


def test_a_block_decides_to_leave_before_its_barrier():
    # the consumers may be in the next phase, and have changed cc.run, when the
    # producer's warp comes out of the grid barrier
    text = _source("sw_project.cu")
    kernel = _body(text, r"cg_ring\(const CgInst")
    after = kernel[kernel.index("cg_grid_sync("):]
    assert "cc." not in after[after.index(";"):]
    sync = _body(text, r"bool cg_grid_sync\([^{]*")
    assert "*run" in sync[sync.index("if (threadIdx.x == 0)"):sync.rindex("__syncthreads()")]


def test_cg_acquires_its_tensor_maps():
    # they lie in a workspace that may have held another grid's maps
    kernel = _body(_source("sw_project.cu"), r"cg_ring\(const CgInst")
    assert 0 <= kernel.find("tmap_acquire(m)") < kernel.index("prefetch_tmap(m)")
    assert kernel.index("prefetch_tmap(m)") < kernel.index("ring_load<")


@pytest.mark.parametrize("name,kernel", [
    ("sw_step_tma.cu", r"step_f32_tma\(const"), ("sw_step_tma.cu", r"step_f64_tma\(const"),
    ("sw_step_tb.cu", r"step_f32_fused2\(const")])
def test_batched_steps_acquire_their_tensor_maps(name, kernel):
    # a batch's maps lie in its table, whose room the next batch uses again
    body = _body(_source(name), kernel)
    at = body.index("if (BATCH && k != acquired)")
    assert at < body.index("tma_load_4d(")
    acquired = set(re.findall(r"tmap_acquire\(([^)]*)\)", body[at:]))
    used = set(re.findall(r"tma_load_4d\([^,]*, ([^,]*),", body))
    assert acquired == used


def test_cg_frees_a_unit_after_its_points():
    # the points' room has no barrier of its own: it is used again on the word
    # of the unit's stage
    tile = _body(_source("sw_project.cu"), r"bool ring_tile\([^{]*")
    walk = _body(tile, r"for \(int j = 0; j < n; j \+= 2[^{]*")
    assert walk.count("release(") == 1
    reads = [m.start() for m in re.finditer(r"finish\(c[01], ap[01], B", walk)]
    assert len(reads) == 2 and "q.points()" in walk[:reads[0]]
    assert walk.index("release(s0)") > max(reads)
