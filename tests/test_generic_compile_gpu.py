"""What a global reduction adds to the compilation of a generated loop, which a user
waits for at the first call: its shuffles and one combination, so well under 60 % of the
same loop without it.  The shortest of six first calls each, in turn."""
import time

import numpy as np
import pytest

pytest.importorskip("torch")  # its NVRTC, where the compilation takes longest

pytestmark = pytest.mark.gpu

BODY = """
inline void %s(double *u, double *du%s) {
  for (int k = 0; k < 4; k++) {
    const double del = du[k];
    u[k] += del;
    du[k] = 0;
    %s
  }
}
"""


def test_reductions_do_not_double_the_compilation(op2):
    n = 1000
    s = op2.op_decl_set(n, "s")
    u = op2.op_decl_dat(s, 4, "double", np.ones((n, 4)), "u")
    du = op2.op_decl_dat(s, 4, "double", np.ones((n, 4)), "du")
    rw = [op2.op_arg_dat(d, -1, op2.OP_ID, 4, "double", op2.OP_RW) for d in (u, du)]
    rms, umax = np.zeros(1), np.full(1, -1e30)
    red = [op2.op_arg_gbl(rms, 1, "double", op2.OP_INC), op2.op_arg_gbl(umax, 1, "double", op2.OP_MAX)]
    for i in range(6):  # registering a source drops what is compiled: before the first call
        op2.register_kernel(f"cmp_plain_{i}", BODY % (f"cmp_plain_{i}", "", ""))
        op2.register_kernel(f"cmp_red_{i}", BODY % (
            f"cmp_red_{i}", ", double *rms, double *umax",
            "*rms += del * del; if (u[k] > *umax) *umax = u[k];"))
    took = {"plain": [], "red": []}
    for i in range(6):
        for kind, args in (("plain", rw), ("red", rw + red)):
            t = time.perf_counter()
            op2.op_par_loop(f"cmp_{kind}_{i}", s, *args)
            took[kind].append(time.perf_counter() - t)
    assert umax[0] == 2.0
    assert min(took["red"]) <= 1.6 * min(took["plain"]), took
