"""The 128-row tcgen05 kernels (blocks of 128 and 256 tokens, head dims 64 and 128) at the edges of their tiles, against
the CPU oracle: live sizes around 0, 1, 64, 128 and the full block, a single tile, odd tile counts, more tiles than any ring
is deep, query and key lengths that differ."""

import pytest
import torch

from oracle import vsa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("be,qb,kb,tk", [(128, 1, 1, 1), (128, 3, 7, 5), (256, 2, 5, 3), (256, 1, 9, 9)])
def test_blocks_of_128_rows_match_the_oracle(be, qb, kb, tk, D, dtype):
    from simple_vsa_b200 import _lib, b200_sparse_attention
    g = torch.Generator().manual_seed(be + 7 * kb + D)
    B, H = 1, 2
    q, dout = (torch.randn(B, H, qb * be, D, generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, H, kb * be, D, generator=g).to(dtype) for _ in range(2))
    sizes = torch.tensor(([be, 1, 0, 64, 127, 128, be - 1, 65, 129 % be] * 2)[:kb])
    # whatever lies in the padding rows must not reach a result
    for x in (k, v):
        x.view(B, H, kb, be, D)[:, :, torch.arange(be)[None, :] >= sizes[:, None]] = float("nan")
    clean = [torch.nan_to_num(x.float(), nan=0.0).to(dtype) for x in (k, v)]
    selected = torch.rand(B, H, qb, kb, generator=g)
    selected[..., 0] = 2.0                                # block 0 is full: every row has a live key
    selected = selected.topk(tk, dim=-1).indices.to(torch.int32)
    want_in = [q.clone().requires_grad_()] + [x.clone().requires_grad_() for x in clean]
    want = O.sparse_attention(*want_in, selected, sizes, be, q_blocks_per_chunk=8)
    want.backward(dout.float())
    leaves = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    out = b200_sparse_attention(*leaves, selected.to(DEV), sizes, block_size=(1, 1, be))
    out.backward(dout.to(DEV))
    assert _lib.device_status() == 0
    # operands, P and dS carry 2^-9 (bf16) or 2^-12 (fp16) each, summed over hundreds of keys: relative 2-norm error near one
    # rounding, far below four of them
    bound = 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    for got, ref in zip([out] + [x.grad for x in leaves], [want] + [x.grad for x in want_in]):
        got, ref = got.detach().float().cpu(), ref.detach().float()
        assert torch.isfinite(got).all()
        assert (got - ref).norm() <= bound * ref.norm()
    dead = torch.arange(be)[None, :] >= sizes[:, None]
    for x in leaves[1:]:
        assert (x.grad.view(B, H, kb, be, D)[:, :, dead.to(DEV)] == 0).all()
