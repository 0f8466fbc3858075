"""The rounding of the weight and bias gradients' sums (op2b_gnn_mlp_dw) over many
rows.  Against FP64 sums of the same bf16 operands the error is no larger than that
of the layer by layer sums, op2b_gemm_bf16 split over the rows and op2b_gnn_colsum:
sums of about as many partial sums of about as many rows, so the errors' norms over
16,384 (128) elements agree to a few (ten) per cent, and 1.25 allows for both.  The
operands have zero mean, and a mean of one standard deviation, where a truncated sum
drifts to one side."""
import ctypes

import pytest

from op2b import gnn as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
W = G.WIDTH


def _ptrs(t, ts):
    return (t * len(ts))(*[x.data_ptr() for x in ts])


@pytest.mark.parametrize("mean", [0.0, 1.0])
@pytest.mark.parametrize("rows,cols", [(300_000, (W,)), (160_000, (W, W)), (635_000, (W, W, W))])
def test_sums_no_further_from_fp64_than_layer_by_layer(op2, rows, cols, mean):
    gen = torch.Generator("cuda").manual_seed(rows + len(cols))
    bf = lambda *s: (torch.randn(*s, device="cuda", generator=gen) + mean).bfloat16()
    st = torch.cuda.current_stream().cuda_stream
    src = [bf(rows if i == 0 else rows // 4, c) for i, c in enumerate(cols)]
    idx = [None] + [torch.randint(rows // 4, (rows,), device="cuda", generator=gen,
                                  dtype=torch.int32) for _ in cols[1:]]
    X = torch.cat([s if r is None else s[r.long()] for s, r in zip(src, idx)], 1).contiguous()
    a0, a1, d0, d1, dy = (bf(rows, W) for _ in range(5))
    parts = (G.op2b_mlp_part * len(cols))(*[(s.data_ptr(), None if r is None else r.data_ptr(), W, W)
                                            for s, r in zip(src, idx)])
    kin = (sum(cols), W, W)
    gw, gb = [torch.zeros(W, k, device="cuda") for k in kin], [torch.zeros(W, device="cuda") for _ in kin]
    G._call("op2b_gnn_mlp_dw", rows, _ptrs(ctypes.c_void_p, [d0, d1, dy]),
            (ctypes.c_long * 3)(W, W, W), W, len(cols), parts, a0.data_ptr(), a1.data_ptr(),
            _ptrs(ctypes.c_void_p, gw), _ptrs(ctypes.c_void_p, gb), st)
    assert G._lib().op2b_gemm_error(0) == 0
    for d, x, g, s, k in zip((d0, d1, dy), (X, a0, a1), gw, gb, kin):
        lw, ls = torch.zeros_like(g), torch.zeros_like(s)
        split = max(1, min(2 * 148 // (k // W), rows // 256))
        G._call("op2b_gemm_bf16", W, k, rows, d.data_ptr(), 1, W, x.data_ptr(), 1, k, lw.data_ptr(),
                k, G.EPI_ATOMIC_F32, None, None, None, 0, split, 0, st)
        G._call("op2b_gnn_colsum", rows, W, d.data_ptr(), W, ls.data_ptr(), st)
        for got, layered, want in ((g, lw, d.double().T @ x.double()), (s, ls, d.double().sum(0))):
            err, was = (float((a.double() - want).norm() / want.norm()) for a in (got, layered))
            print("rows %d k %d mean %g: error %.3g, layer by layer %.3g" % (rows, k, mean, err, was))
            assert err <= 1.25 * was


def test_an_infinite_gradient_stays_infinite(op2):
    rows, st = 20_000, torch.cuda.current_stream().cuda_stream
    x, a0, a1, d0, d1, dy = (torch.ones(rows, W, device="cuda").bfloat16() for _ in range(6))
    d1[5, 3] = float("inf")
    gw, gb = [torch.zeros(W, W, device="cuda") for _ in range(3)], [torch.zeros(W, device="cuda") for _ in range(3)]
    parts = (G.op2b_mlp_part * 1)((x.data_ptr(), None, W, W))
    G._call("op2b_gnn_mlp_dw", rows, _ptrs(ctypes.c_void_p, [d0, d1, dy]),
            (ctypes.c_long * 3)(W, W, W), W, 1, parts, a0.data_ptr(), a1.data_ptr(),
            _ptrs(ctypes.c_void_p, gw), _ptrs(ctypes.c_void_p, gb), st)
    want = torch.full((W,), float(rows), device="cuda")
    want[3] = float("inf")
    assert torch.equal(gb[1], want) and torch.equal(gw[1], want[:, None].expand(W, W))
    assert torch.equal(gb[0], torch.full_like(want, rows))
