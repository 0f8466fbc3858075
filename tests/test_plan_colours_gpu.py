"""Greedy block colours of the execution plan against first-fit in block order
on the host: more than 32 colours (several passes), partial last blocks, more
targets a block than are loaded ahead (2048), one block, and the blkmap that
groups the blocks by colour in block order."""
import numpy as np
import pytest

from op2b import lib as L
from op2b import mesh as M

pytestmark = pytest.mark.gpu


def first_fit(targets, part, n):
    """Colour per block; targets: (n, k) ids each element increments."""
    used = {}
    out = []
    for b in range(0, n, part):
        t = np.unique(targets[b:b + part])
        mask = 0
        for v in t:
            mask |= used.get(int(v), 0)
        c = 0
        while mask >> c & 1:
            c += 1
        out.append(c)
        for v in t:
            used[int(v)] = used.get(int(v), 0) | (1 << c)
    return np.array(out)


@pytest.mark.parametrize("I,J,permute", [(5, 3, True), (61, 37, False), (120, 60, True)])
@pytest.mark.parametrize("part,slots", [(64, 2), (256, 2), (256, 4), (1024, 2), (1024, 4)])
def test_block_colours_are_first_fit(op2, I, J, permute, part, slots):
    m = M.channel_bump(I, J, seed=5, permute=permute)
    nodes, cells = op2.op_decl_set(m.nnode, "nodes"), op2.op_decl_set(m.ncell, "cells")
    pcell = op2.op_decl_map(cells, nodes, 4, m.cell, "pcell")
    d = op2.op_decl_dat(nodes, 1, "double", None, "d")
    args = [op2.op_arg_dat(d, k, pcell, 1, "double", L.OP_INC) for k in range(slots)]
    p = L.op_plan_get_stage("colours", cells, part, args, [0] * slots, L.OP_STAGE_INC)
    a = L.plan_arrays(p)
    col = first_fit(m.cell[:, :slots], part, m.ncell)
    assert a["ncolors"] == col.max() + 1
    assert np.array_equal(a["ncolblk"], np.bincount(col))
    assert np.array_equal(a["blkmap"], np.argsort(col, kind="stable"))
    if (I, part) == (120, 64):
        assert a["ncolors"] > 32
