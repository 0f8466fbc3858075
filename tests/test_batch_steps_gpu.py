"""The batch engine's fused step kernels (res_calc with bres_calc, update with
save_soln and the next adt_calc) against the plain loops, dat by dat."""
import numpy as np
import pytest

from op2b import mesh as M
from op2b.airfoil import Airfoil
from op2b.batch import AirfoilBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [(1,), (3, 2)])
@pytest.mark.parametrize("part_size", [0, 300])
def test_fp64_batch_leaves_every_dat_as_the_plain_loops_do(op2, runs, part_size):
    """One renumbered instance: q, qold, adt and res after the runs are those of
    the plain loops bit for bit (the same increments in the same order), also
    when the caller reads them between two runs, and rms to rounding."""
    spec = dict(I=61, J=37, mach=0.45, alpha=2.0, bump=0.05, seed=3)
    b = AirfoilBatch([spec], fp32=False)
    for k, v in (("tol", 0.0), ("stall_window", 1e6)):
        b.set(k, v)
    if part_size:
        b.set("part_size", part_size)
    for n in runs:
        b.run(n)
        got = [op2.op_fetch_data(d) for d in (b.d64.p_q, b.d64.p_qold, b.d64.p_adt, b.d64.p_res)]
    rms = b.stats()["rms_last"][0]
    b.close()
    op2.op_exit()
    op2.op_init()
    app = Airfoil(M.channel_bump(61, 37, seed=3, bump=0.05),
                  M.airfoil_constants(mach=0.45, alpha_deg=2.0))
    app.renumber()
    hist = app.iterate(sum(runs))
    want = app.fetch()
    for g, k in zip(got, ("q", "qold", "adt", "res")):
        assert np.array_equal(g.reshape(want[k].shape), want[k]), k
    assert abs(rms / hist[-1][0] - 1) < 1e-12


def test_batch_survives_another_meshs_renumbering(op2):
    """op_renumber drops every mesh's cached records; a batch finds its own again."""
    spec = dict(I=24, J=12, mach=0.5, alpha=1.0, bump=0.05, seed=1)
    b = AirfoilBatch([spec], fp32=False)
    b.run(2)
    other = Airfoil(M.channel_bump(40, 20, seed=2))
    other.renumber()
    other.iterate(1)
    b.run(3)
    got = b.q_instance(0)
    b.close()
    c = AirfoilBatch([spec], fp32=False)
    c.run(5)
    assert np.array_equal(got, c.q_instance(0))
    c.close()
