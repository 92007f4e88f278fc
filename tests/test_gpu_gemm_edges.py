"""The GEMM's two epilogues: whole sectors per lane where the output's rows
start on 32-byte boundaries and the slab of 32 columns is whole, else through
shared memory.  Row lengths and M on both sides of each line, against a
PyTorch fp32 matmul (products are exact in fp32; 1e-4 of the largest value
plus 1e-3 for the order of summation, as at the other sizes)."""
import pytest

from m6502.mlp import gemm_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 31, 33, 127, 129])
@pytest.mark.parametrize("N", [1, 8, 31, 32, 33, 40, 201, 256, 264, 511])
def test_gemm_at_row_ends(engine, M, N):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    a = torch.randn((M, 192), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((N, 192), generator=g, device="cuda").to(torch.bfloat16)
    ref = a.float() @ b.float().T
    c = gemm_bf16(engine, a, b)
    assert (c - ref).abs().max().item() <= 1e-4 * ref.abs().max().item() + 1e-3
    big = torch.full((M * N + 1,), 7.0, device="cuda")     # an output 4 bytes off every boundary; nothing past it is written
    import ctypes
    from m6502 import _lib
    engine.order_after_torch()
    rc = _lib.lib().m6502_gemm_bf16(engine._ctx, M, N, 192, ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()),
                                    ctypes.c_void_p(big.data_ptr() + 4))
    assert rc == 0 and big[0].item() == 7.0
    assert torch.equal(big[1:].view(M, N), c)
