"""The batch engine's paths that the FP64 step test does not take, against the plain
loops (the same increments in the same order: bit for bit): FP32 storage dat by dat, the
first FP64 step after a promotion, and res_calc and bres_calc as loops of their own, on a
mesh whose boundary edges cannot be linked into the corner records."""
import numpy as np
import pytest

from op2b import lib as L
from op2b import mesh as M
from op2b.airfoil import Airfoil
from op2b.batch import AirfoilBatch
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SPEC = dict(I=61, J=37, mach=0.45, alpha=2.0, bump=0.05, seed=3)
CONSTS = dict(mach=0.45, alpha_deg=2.0)


def _mesh():
    return M.channel_bump(61, 37, seed=3, bump=0.05)


def _batch(fp32, meshes=None, **keys):
    b = AirfoilBatch([SPEC], fp32=fp32, meshes=meshes)
    for k, v in dict(dict(tol=0.0, stall_window=1e6), **keys).items():
        b.set(k, v)
    return b


def _fetch(op2, d):
    return [op2.op_fetch_data(x) for x in (d.p_q, d.p_qold, d.p_adt, d.p_res)]


def _plain(op2, iters, mesh=None, **kw):
    """The loops on the same mesh, renumbered alike, in a session of their own."""
    op2.op_exit()
    op2.op_init()
    app = Airfoil(mesh or _mesh(), M.airfoil_constants(**CONSTS), **kw)
    app.renumber()
    hist = app.iterate(iters)
    return app.fetch(), hist[-1][0]


def _equal(got, want):
    for g, k in zip(got, ("q", "qold", "adt", "res")):
        assert np.array_equal(g.reshape(want[k].shape), want[k]), k


@pytest.mark.parametrize("runs", [(1,), (3, 2)])
def test_fp32_batch_leaves_every_dat_as_the_float_loops_do(op2, runs):
    b = _batch(True, promote_tol=0.0)
    for n in runs:
        b.run(n)
    got, rms = _fetch(op2, b.d32), b.stats()["rms_last"][0]
    b.close()
    want, last = _plain(op2, sum(runs), dtype=np.float32)
    _equal(got, want)
    assert abs(rms / last - 1) < 1e-12


@pytest.mark.parametrize("runs", [(1, 1), (2,), (1, 2)])
def test_first_fp64_step_after_a_promotion(op2, runs):
    """promote_tol 2: an instance is promoted after its first iteration."""
    b = _batch(True, promote_tol=2.0)
    for n in runs:
        b.run(n)
    got, st = _fetch(op2, b.d64), b.stats()
    assert list(st["iters32"]) == [1] and list(st["iters"]) == [sum(runs)]
    b.close()
    op2.op_exit()
    op2.op_init()
    b = _batch(True, promote_tol=2.0)
    b.run(1)
    q32 = b.q_all("fp32").astype(np.float64)  # declared order
    b.close()
    want, _ = _plain(op2, sum(runs) - 1, q0=q32)
    _equal(got, want)


@pytest.mark.parametrize("runs", [(1,), (3, 2)])
def test_boundary_edges_that_cannot_be_linked(op2, runs):
    """A boundary edge given twice: its cell has five edges, one more than slots."""
    m = _mesh()
    again = lambda a: np.concatenate([a, a[7:8]])
    m.bedge, m.becell, m.bound = again(m.bedge), again(m.becell), again(m.bound)
    b = _batch(False, meshes=[m])
    for n in runs:
        before = L.load().op2b_kernel_launches()
        b.run(n)
        # adt_calc once, three loops a step, the convergence
        assert L.load().op2b_kernel_launches() - before == 1 + 7 * n
    got, q = _fetch(op2, b.d64), b.q_all()
    b.close()
    want, _ = _plain(op2, sum(runs), mesh=m)
    _equal(got, want)
    st, _, _, _ = O.airfoil_run(m, M.airfoil_constants(**CONSTS), sum(runs))
    assert np.all(np.abs(q - st.q).max(axis=0) <= 1e-12 * np.abs(st.q).max(axis=0))
