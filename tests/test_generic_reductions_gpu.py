"""Global reductions of generated loops: blocks' partials combined by the last
block and read from the mapped page, against numpy, at set sizes on both sides
of a warp, a block and the grid's bound (148 x 8 blocks), for every type and
access together, several components, empty sets and more entries than the
block reduction takes (64: those keep the atomics).  Sums: each side rounds at most
once an addition, 1e-12 of the magnitudes' sum in double, 1e-5 in float; minima,
maxima and integers exactly."""
import numpy as np
import pytest

from op2b import lib as L

pytestmark = pytest.mark.gpu

KERNEL = """
inline void redk_%(d)d(const double *a, const float *f, const int *i, double *s, double *mn,
                       float *fs, float *fx, int *is, int *ix) {
  for (int k = 0; k < %(d)d; k++) {
    s[k] += (k + 1) * a[0];
    if (a[0] - k < mn[k]) mn[k] = a[0] - k;
  }
  fs[0] += f[0];
  if (f[0] > fx[0]) fx[0] = f[0];
  is[0] += i[0];
  if (i[0] > ix[0]) ix[0] = i[0];
}
"""


@pytest.mark.parametrize("n", [0, 1, 31, 33, 255, 257, 148 * 8 * 256 - 1, 148 * 8 * 256 + 1, 700001])
@pytest.mark.parametrize("d", [1, 5, 40])
def test_reductions_of_every_type(op2, n, d):
    if d > 5 and n > 300:
        pytest.skip("the many-entry form at the small sizes only")
    op2.register_kernel(f"redk_{d}", KERNEL % dict(d=d))
    rng = np.random.default_rng(n + d)
    s = op2.op_decl_set(n, "s")
    a, f = rng.standard_normal((n, 1)), rng.standard_normal((n, 1)).astype(np.float32)
    i = rng.integers(-1000, 1000, (n, 1)).astype(np.int32)
    A = lambda dat, t: op2.op_arg_dat(dat, -1, op2.OP_ID, 1, t, op2.OP_READ)
    pa, pf, pi = (op2.op_decl_dat(s, 1, t, v, nm) for t, v, nm in
                  (("double", a, "a"), ("float", f, "f"), ("int", i, "i")))
    for start in (0.0, 2.5):  # the caller's values count
        sd, mn = np.full(d, start), np.full(d, start - 0.5)
        fs, fx = np.full(1, start, np.float32), np.full(1, start, np.float32)
        si, ix = np.full(1, 3, np.int32), np.full(1, -5, np.int32)
        op2.op_par_loop(f"redk_{d}", s, A(pa, "double"), A(pf, "float"), A(pi, "int"),
                        op2.op_arg_gbl(sd, d, "double", op2.OP_INC),
                        op2.op_arg_gbl(mn, d, "double", op2.OP_MIN),
                        op2.op_arg_gbl(fs, 1, "float", op2.OP_INC),
                        op2.op_arg_gbl(fx, 1, "float", op2.OP_MAX),
                        op2.op_arg_gbl(si, 1, "int", op2.OP_INC),
                        op2.op_arg_gbl(ix, 1, "int", op2.OP_MAX))
        k = np.arange(d)
        assert np.all(np.abs(sd - start - (k + 1) * a.sum()) <= 1e-12 * (k + 1) *
                      (np.abs(a).sum() + abs(start)))
        assert np.array_equal(mn, np.minimum(start - 0.5, a.min() - k) if n else
                              np.full(d, start - 0.5))
        assert abs(float(fs[0]) - start - f.astype(np.float64).sum()) <= 1e-5 * (
            np.abs(f).sum() + abs(start))
        assert fx[0] == max(np.float32(start), f.max() if n else np.float32(start))
        assert si[0] == 3 + i.sum() and ix[0] == max(-5, i.max() if n else -5)


def test_reduction_is_the_same_every_run(op2):
    op2.register_kernel("redk_1", KERNEL % dict(d=1))
    n = 300001
    rng = np.random.default_rng(0)
    s = op2.op_decl_set(n, "s")
    pa = op2.op_decl_dat(s, 1, "double", rng.standard_normal((n, 1)), "a")
    pf = op2.op_decl_dat(s, 1, "float", rng.standard_normal((n, 1)).astype(np.float32), "f")
    pi = op2.op_decl_dat(s, 1, "int", np.ones((n, 1), np.int32), "i")
    A = lambda dat, t: op2.op_arg_dat(dat, -1, op2.OP_ID, 1, t, op2.OP_READ)
    got = []
    for _ in range(4):
        out = [np.zeros(1), np.zeros(1), np.zeros(1, np.float32), np.zeros(1, np.float32),
               np.zeros(1, np.int32), np.zeros(1, np.int32)]
        acc = [L.OP_INC, L.OP_MIN, L.OP_INC, L.OP_MAX, L.OP_INC, L.OP_MAX]
        types = ["double", "double", "float", "float", "int", "int"]
        op2.op_par_loop("redk_1", s, A(pa, "double"), A(pf, "float"), A(pi, "int"),
                        *[op2.op_arg_gbl(o, 1, t, c) for o, t, c in zip(out, types, acc)])
        got.append([o.tobytes() for o in out])
    assert all(g == got[0] for g in got)
