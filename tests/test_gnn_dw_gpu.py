"""The weight gradients of one MLP (op2b_gnn_mlp_dw) over the ways its operands
arrive: rows of at least 64 columns by TMA (the second box of 64 columns partly or
wholly outside), narrower and indexed ones by 16-byte copies, both in one layer.
Against FP64 sums of the same bf16 operands: FP32 sums over the rows in another
grouping are within 1e-5 of the gradient's norm (rows x 2^-24 at worst)."""
import ctypes

import pytest

from op2b import gnn as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
W = G.WIDTH


def _ptrs(t, ts):
    return (t * len(ts))(*[x.data_ptr() for x in ts])


@pytest.mark.parametrize("rows", [1, 63, 65, 148 * 64 * 4 + 5])
@pytest.mark.parametrize("cols,indexed,nout", [
    ((56,), (0,), 16), ((64,), (0,), W), ((72,), (0,), 8), ((120,), (0,), W),
    ((W, W), (0, 0), W), ((W, W, W), (0, 1, 0), W), ((W, W, W), (0, 0, 1), 16),
])
def test_weight_gradients(op2, rows, cols, indexed, nout):
    gen = torch.Generator("cuda").manual_seed(rows + sum(cols) + nout)
    bf = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    nsrc = max(rows // 3, 1)
    src = [bf(nsrc if i else rows, c + 8) for i, c in zip(indexed, cols)]  # rows with a pad
    idx = [torch.randint(nsrc, (rows,), device="cuda", generator=gen, dtype=torch.int32) if i
           else None for i in indexed]
    X = torch.cat([(s if r is None else s[r.long()])[:, :c] for s, r, c in zip(src, idx, cols)], 1)
    a0, a1, d0, d1 = (bf(rows, W) for _ in range(4))
    dy = bf(rows, nout)
    parts = (G.op2b_mlp_part * len(cols))(*[
        (s.data_ptr(), None if r is None else r.data_ptr(), c + 8, c)
        for s, r, c in zip(src, idx, cols)])
    gw = [torch.ones(o, k, device="cuda") for k, o in ((sum(cols), W), (W, W), (W, nout))]
    gb = [torch.ones(o, device="cuda") for o in (W, W, nout)]
    G._call("op2b_gnn_mlp_dw", rows, _ptrs(ctypes.c_void_p, [d0, d1, dy]),
            (ctypes.c_long * 3)(W, W, nout), nout, len(cols), parts, a0.data_ptr(), a1.data_ptr(),
            _ptrs(ctypes.c_void_p, gw), _ptrs(ctypes.c_void_p, gb),
            torch.cuda.current_stream().cuda_stream)
    for d, x, g, s in zip((d0, d1, dy), (X, a0, a1), gw, gb):
        for a, r in ((g, d.double().T @ x.double()), (s, d.double().sum(0))):
            err = float((a.double() - 1.0 - r).norm())
            assert err <= 1e-5 * max(float(r.norm()), float(r.numel()) ** 0.5), err
    assert G._lib().op2b_gemm_error(0) == 0
