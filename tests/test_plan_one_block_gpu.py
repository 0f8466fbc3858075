"""A plan of one block: one colour, found without the colouring's sweep over the block's
targets (of OP_COLOR2 the whole set, more pairs of argument and element than an int
counts on the largest).  Against a plan of two blocks, which has it."""
import pytest

from op2b import lib as L
from op2b import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_one_block_has_one_colour_and_no_sweep(op2, mode):
    m = M.channel_bump(40, 25, seed=4)
    nodes, cells = op2.op_decl_set(m.nnode, "nodes"), op2.op_decl_set(m.ncell, "cells")
    pcell = op2.op_decl_map(cells, nodes, 4, m.cell, "pcell")
    d = op2.op_decl_dat(nodes, 1, "double", None, "d")
    args = [op2.op_arg_dat(d, k, pcell, 1, "double", L.OP_INC) for k in range(2)]
    op2.set_option("plan_mode", mode)
    launches = {}
    for what, part, staging in (("two", 512, L.OP_STAGE_INC), ("one", 1024, L.OP_STAGE_INC),
                                ("flat", 0, L.OP_COLOR2)):
        before = L.load().op2b_kernel_launches()
        p = L.op_plan_get_stage(what, cells, part, args, [0, 0], staging)
        launches[what] = L.load().op2b_kernel_launches() - before
        a = L.plan_arrays(p)
        nblocks = 2 if what == "two" else 1
        assert p.contents.nblocks == nblocks and L.plan_validate(p)[0] == 0
        if what == "one":
            assert a["ncolors"] == 1 and list(a["ncolblk"]) == [1] and list(a["blkmap"]) == [0]
        if what == "flat":
            assert a["ncolblk"][0] == 1 and a["blkmap"][0] == 0
    op2.set_option("plan_mode", 0)
    if mode == 0:
        assert launches["one"] == launches["two"] - 1
