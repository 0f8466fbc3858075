"""Plans' device arrays may be read on a stream of the caller's: releasing the plans, or
a renumbering that drops them, waits for it."""
import pytest

from op2b import lib as L
from op2b import mesh as M

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("by", ["release_all", "renumber"])
def test_release_waits_for_the_callers_stream(op2, by):
    m = M.channel_bump(61, 37, seed=2)
    nodes, cells = op2.op_decl_set(m.nnode, "nodes"), op2.op_decl_set(m.ncell, "cells")
    pcell = op2.op_decl_map(cells, nodes, 4, m.cell, "pcell")
    edges = op2.op_decl_set(m.nedge, "edges")
    pecell = op2.op_decl_map(edges, cells, 2, m.ecell, "pecell")
    d = op2.op_decl_dat(nodes, 1, "double", None, "d")
    args = [op2.op_arg_dat(d, k, pcell, 1, "double", L.OP_INC) for k in range(2)]
    if by == "renumber":
        op2.op_renumber(pecell, stats=False)  # what a first one sets up is not what is tested
    assert L.op_plan_get_stage("release", cells, 256, args, [0, 0], L.OP_STAGE_INC)
    mine = torch.cuda.Stream()
    with torch.cuda.stream(mine):
        torch.cuda._sleep(400_000_000)  # about 0.2 s, in place of a kernel that reads the plan
    assert not mine.query()
    if by == "release_all":
        L.load().op2b_plan_release_all()
    else:
        op2.op_renumber(pecell, stats=False)
    assert mine.query()
