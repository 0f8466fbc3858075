"""Coloured loops whose colours run in one cluster's launch, against numpy:
read-modify-write through a map whose targets are shared by many elements
(integer values, so every order is exact), at sizes on both sides of a block,
of eight blocks a colour, and of the size that keeps a launch a colour."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNEL = """
inline void clus_add(double *a, double *b, const double *w) {
  a[0] = a[0] + w[0];
  b[0] = b[0] + 2 * w[0];
}
"""


@pytest.mark.parametrize("n", [1, 2, 255, 257, 3000, 16384, 16385])
@pytest.mark.parametrize("targets", [2, 61, 5000])
def test_coloured_read_write(op2, n, targets):
    if targets < 61 and n > 300:
        pytest.skip("as many colours as elements")
    op2.register_kernel("clus_add", KERNEL)
    rng = np.random.default_rng(n + targets)
    a = rng.integers(targets, size=n)
    b = (a + 1 + rng.integers(targets - 1, size=n)) % targets
    m = np.stack([a, b], 1).astype(np.int32)
    w = rng.integers(-50, 50, (n, 1)).astype(np.float64)
    e, t = op2.op_decl_set(n, "e"), op2.op_decl_set(targets, "t")
    pm = op2.op_decl_map(e, t, 2, m, "m")
    pt = op2.op_decl_dat(t, 1, "double", None, "v")
    pw = op2.op_decl_dat(e, 1, "double", w, "w")
    for _ in range(3):
        op2.op_par_loop("clus_add", e, op2.op_arg_dat(pt, 0, pm, 1, "double", op2.OP_RW),
                        op2.op_arg_dat(pt, 1, pm, 1, "double", op2.OP_RW),
                        op2.op_arg_dat(pw, -1, op2.OP_ID, 1, "double", op2.OP_READ))
    ref = np.zeros(targets)
    np.add.at(ref, a, 3 * w[:, 0])
    np.add.at(ref, b, 6 * w[:, 0])
    assert np.array_equal(op2.op_fetch_data(pt)[:, 0], ref)
