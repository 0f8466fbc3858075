"""The tensor-core product's operand R (residual, or SiLU' argument): fetched by
TMA where its rows are whole 16-byte pieces, by each lane otherwise.  Both give
the bits of the one-tile kernel (engine 0 with gemm_tma off): the K order and
the epilogue's arithmetic are the same."""
import pytest
import torch

from op2b import gnn as G
from op2b import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epi", [G.EPI_BIAS_BF16, G.EPI_SILU_GRAD_BF16])
@pytest.mark.parametrize("rows,n,k,shift", [
    (1, 8, 8, 0), (33, 40, 64, 0), (129, 136, 72, 0),
    (128 * 148 * 2 + 37, 128, 128, 0),   # more than one tile a CTA, a ragged last one
    (128 * 148 + 1, 264, 16, 0),         # three column tiles, the last of 8 columns
    (128 * 148 * 2 + 37, 128, 128, 4),   # R off the 16-byte grid: read by the lanes
])
def test_row_operand_gives_the_same_bits(epi, rows, n, k, shift):
    L.op_init()
    torch.manual_seed(rows + n)
    dev = "cuda"
    a = torch.randn(rows, k, device=dev).bfloat16()
    b = torch.randn(n, k, device=dev).bfloat16()
    bias = torch.randn(n, device=dev) if epi == G.EPI_BIAS_BF16 else None
    ldr = n + 8
    r = torch.randn(rows * ldr + shift, device=dev).bfloat16()
    out = []
    for engine in (2, 0):
        if engine == 0:
            old = L.get_option("gemm_tma")
            L.set_option("gemm_tma", 0)
        c = torch.full((rows, n + 8), 7.0, device=dev).bfloat16()
        G._call("op2b_gemm_bf16", rows, n, k, a.data_ptr(), k, 1, b.data_ptr(), k, 1,
                c.data_ptr(), n + 8, epi, bias.data_ptr() if bias is not None else None, None,
                r.data_ptr() + 2 * shift, ldr, 1, engine, torch.cuda.current_stream().cuda_stream)
        if engine == 0:
            L.set_option("gemm_tma", old)
        out.append(c)
    torch.cuda.synchronize()
    assert torch.equal(out[0].view(torch.int16), out[1].view(torch.int16))
    assert bool((out[0][:, n:] == 7.0).all())
