"""The one-kernel MLPs of the graph network (op2b_gnn_mlp, _backward, _dw)
against the same MLP layer by layer on the register-staged product
(op2b_gemm_bf16, engine 0): the MMAs run over K in the same order and every
value is rounded to bf16 at the same point, so outputs, kept activations and
input gradients are equal bit for bit.  Weight and bias gradients are FP32
sums over the rows in another grouping: within 1e-5 of their norm (rows x 2^-24
at worst, far less for random signs).  Row counts sit on both sides of a tile
(128), of the dW block (64) and of one tile an SM."""
import ctypes

import numpy as np
import pytest

from op2b import gnn as G
from op2b import lib as L
from op2b import mesh as M

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
W = G.WIDTH


def _gemm(M_, N, K, A, a_m, a_k, B, b_n, b_k, C, ldc, epi, bias=None, Z=None, R=None, ldr=0):
    ptr = lambda t: None if t is None else t.data_ptr()
    G._call("op2b_gemm_bf16", M_, N, K, ptr(A), a_m, a_k, ptr(B), b_n, b_k, ptr(C), ldc, epi,
            ptr(bias), ptr(Z), ptr(R), ldr, 1, 0, torch.cuda.current_stream().cuda_stream)


def _ptrs(t, ts):
    return (t * len(ts))(*[x.data_ptr() if torch.is_tensor(x) else x for x in ts])


CASES = [(rows, cols, nout) for rows in (1, 63, 65, 127, 128, 129, 300, 148 * 128 + 1, 60000)
         for cols, nout in (((8,), W), ((16,), W), ((64,), W), ((W,), 8), ((W, W), W),
                            ((W, W, W), W)) if rows < 1000 or cols != (64,)]


@pytest.mark.parametrize("rows,cols,nout", CASES)
def test_mlp_kernels_equal_layer_by_layer(op2, rows, cols, nout):
    gen = torch.Generator("cuda").manual_seed(rows + sum(cols) + nout)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    bf = lambda t: t.to(torch.bfloat16)
    st = torch.cuda.current_stream().cuda_stream
    kin, nsrc = sum(cols), max(rows // 3, 1)
    src = [bf(rnd(rows if i == 0 else nsrc, c)) for i, c in enumerate(cols)]
    idx = [None] + [torch.randint(nsrc, (rows,), device="cuda", generator=gen, dtype=torch.int32)
                    for _ in cols[1:]]
    X = torch.cat([s if r is None else s[r.long()] for s, r in zip(src, idx)], 1).contiguous()
    w = [bf(rnd(o, k) / k ** 0.5) for k, o in ((kin, W), (W, W), (W, nout))]
    b = [0.2 * rnd(o) for o in (W, W, nout)]
    res = src[0] if cols[0] == W and nout == W else None
    # layer by layer
    z0, a0, z1, a1 = (torch.zeros(rows, W, dtype=torch.bfloat16, device="cuda") for _ in range(4))
    y = torch.zeros(rows, nout, dtype=torch.bfloat16 if nout == W else torch.float32,
                    device="cuda")
    _gemm(rows, W, kin, X, kin, 1, w[0], kin, 1, a0, W, G.EPI_BIAS_SILU_BF16, b[0], z0)
    _gemm(rows, W, W, a0, W, 1, w[1], W, 1, a1, W, G.EPI_BIAS_SILU_BF16, b[1], z1)
    _gemm(rows, nout, W, a1, W, 1, w[2], W, 1, y, nout,
          G.EPI_BIAS_BF16 if nout == W else G.EPI_STORE_F32, b[2], None, res, W)
    # one kernel, with and without the kept activations
    parts = (G.op2b_mlp_part * len(cols))(*[
        (s.data_ptr(), None if r is None else r.data_ptr(), c, c)
        for s, r, c in zip(src, idx, cols)])
    for keep in (True, False):
        kept = [torch.full_like(z0, 7.0) for _ in range(4)]
        out = torch.full_like(y, 7.0)
        G._call("op2b_gnn_mlp", rows, len(cols), parts, _ptrs(ctypes.c_void_p, w),
                _ptrs(ctypes.c_void_p, b), nout, None if res is None else res.data_ptr(), W,
                out.data_ptr(), nout, *([t.data_ptr() for t in kept] if keep else [None] * 4), st)
        assert torch.equal(out, y)
        for got, want in zip(kept, (z0, a0, z1, a1)):
            assert torch.equal(got, want) if keep else bool((got == 7.0).all())
    # backward
    dy = bf(rnd(rows, nout))
    d1, d0, e1, e0 = (torch.zeros_like(z0) for _ in range(4))
    _gemm(rows, W, nout, dy, nout, 1, w[2], 1, W, d1, W, G.EPI_SILU_GRAD_BF16, R=z1, ldr=W)
    _gemm(rows, W, W, d1, W, 1, w[1], 1, W, d0, W, G.EPI_SILU_GRAD_BF16, R=z0, ldr=W)
    np_ = kin // W
    dx = torch.zeros(rows, kin, device="cuda")
    _gemm(rows, kin, W, d0, W, 1, w[0], 1, kin, dx, kin, G.EPI_STORE_F32)
    base = rnd(rows, W)
    got = [base.clone()] + [torch.full((rows, W), 7.0, device="cuda") for _ in range(2)]
    G._call("op2b_gnn_mlp_backward", rows, dy.data_ptr(), nout, nout, _ptrs(ctypes.c_void_p, w),
            kin, z0.data_ptr(), z1.data_ptr(), e0.data_ptr(), e1.data_ptr(), np_,
            _ptrs(ctypes.c_void_p, got), (ctypes.c_long * 3)(W, W, W), (ctypes.c_int * 3)(1, 0, 0),
            st)
    assert torch.equal(e1, d1) and torch.equal(e0, d0)
    for p in range(np_):
        want = dx[:, p * W:(p + 1) * W]
        assert torch.equal(got[p], base + want if p == 0 else want)
    # weight and bias gradients, added to what is there
    gw = [torch.ones(o, k, device="cuda") for k, o in ((kin, W), (W, W), (W, nout))]
    gb = [torch.ones(o, device="cuda") for o in (W, W, nout)]
    G._call("op2b_gnn_mlp_dw", rows, _ptrs(ctypes.c_void_p, [d0, d1, dy]),
            (ctypes.c_long * 3)(W, W, nout), nout, len(cols), parts, a0.data_ptr(), a1.data_ptr(),
            _ptrs(ctypes.c_void_p, gw), _ptrs(ctypes.c_void_p, gb), st)
    for d, x, g, s in zip((d0, d1, dy), (X, a0, a1), gw, gb):
        for a, r in ((g, d.double().T @ x.double()), (s, d.double().sum(0))):
            err = float((a.double() - 1.0 - r).norm())
            assert err <= 1e-5 * max(float(r.norm()), float(r.numel()) ** 0.5), err
    torch.cuda.synchronize()
    assert G._lib().op2b_gemm_error(1) == 0


def test_mlp_entries_refuse_what_they_cannot_run(op2):
    t = torch.zeros(256, 3 * W, dtype=torch.bfloat16, device="cuda")
    f = torch.zeros(W, device="cuda")
    w, b = _ptrs(ctypes.c_void_p, [t] * 3), _ptrs(ctypes.c_void_p, [f] * 3)

    def call(parts, nout=W, y=t.data_ptr()):
        arr = (G.op2b_mlp_part * len(parts))(*parts)
        return G._lib().op2b_gnn_mlp(128, len(parts), arr, w, b, nout, None, 0, y, W, None, None,
                                     None, None, None)
    p = t.data_ptr()
    assert call([(p, None, W, 72)]) == -1                      # neither 8..64 nor 128 columns
    assert call([(p + 2, None, W, W)]) == -1                   # unaligned rows
    assert call([(p, p, W, W)]) == -1                          # an indexed first part
    assert call([(p, None, W, W), (p, None, W, 64)]) == -1     # a short later part
    assert call([(p, None, W, W)], nout=24) == -1
    assert call([(p, None, W, W)], y=p + 16) == -1             # rows not 32-byte aligned


@pytest.mark.parametrize("I,J,steps,copies", [(4, 3, 2, 1), (24, 12, 3, 2), (61, 37, 8, 1)])
def test_network_equals_layer_by_layer(op2, I, J, steps, copies):
    m = M.channel_bump(I, J, seed=3, bump=0.07)
    g1 = G.cell_graph(m)
    g = G.replicate_graph(g1, copies)
    ni = torch.from_numpy(G.node_features(m, 0.5, 2.0, 0.07)).cuda().repeat(copies, 1)
    ei = torch.from_numpy(G.edge_features(m, g1)).cuda().repeat(copies, 1)
    tg = torch.from_numpy(np.random.default_rng(1).standard_normal((g["N"], 4)).astype(
        np.float32)).cuda()
    got = []
    for fused in (True, False):
        net = G.GraphNet(steps=steps, seed=4)
        net.gemm_tma = fused
        dg = net.upload_graph(g)
        infer = net.forward(dg, ni, ei, train=False).clone()
        net.loss_grad(dg, ni, ei, tg)
        ws = net.workspace(g["N"], g["E"], True)
        assert torch.equal(infer, ws["out"])
        got.append((ws["out"].clone(), ws["dE"].clone(), ws["dH"].clone(), net.g.clone()))
    a, b = got
    assert all(torch.equal(x, y) for x, y in zip(a[:3], b[:3]))
    assert float((a[3] - b[3]).norm()) <= 1e-5 * float(b[3].norm())
    assert G._lib().op2b_gemm_error(1) == 0
