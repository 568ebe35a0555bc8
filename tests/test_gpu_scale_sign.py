"""`sm_scale` is any number: negative and zero scales give the output and the gradients of the formula on every kernel family."""

import pytest
import torch

from oracle import vsa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("scale", [-0.11, 0.0])
@pytest.mark.parametrize("be,D,dtype,nb,tk", [(64, 128, torch.bfloat16, 6, 4), (128, 128, torch.float16, 6, 4), (256, 128, torch.bfloat16, 6, 4),
                                              (64, 64, torch.float16, 6, 4), (128, 64, torch.bfloat16, 6, 4), (256, 64, torch.float16, 6, 4),
                                              (64, 64, torch.float16, 10, 9), (64, 64, torch.bfloat16, 10, 8),     # 64-row tcgen05 in every pass
                                              (64, 64, torch.float32, 6, 4), (8, 16, torch.float32, 6, 4)])
def test_negative_and_zero_scale_match_the_oracle(be, D, dtype, nb, tk, scale):
    from simple_vsa_b200 import _lib, b200_sparse_attention
    g = torch.Generator().manual_seed(be + D)
    B, H = 1, 2
    if tk >= 8:
        assert all(_lib.lib.vsa_sparse_pass_kernels(p, B * H, nb * be, D, be, tk, _lib.VSA_F16) == 2 for p in range(3))
    q, k, v, dout = (torch.randn(B, H, nb * be, D, generator=g).to(dtype) for _ in range(4))
    sizes = torch.tensor(([be, be - 1, be, be // 2 + 1, be, 3] * 2)[:nb])
    selected = torch.rand(B, H, nb, nb, generator=g).topk(tk, dim=-1).indices.to(torch.int32)
    want_in = [x.clone().requires_grad_() for x in (q, k, v)]
    want = O.sparse_attention(*want_in, selected, sizes, be, scale)
    want.backward(dout.float())
    leaves = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    out = b200_sparse_attention(*leaves, selected.to(DEV), sizes, block_size=(1, 1, be), sm_scale=scale)
    out.backward(dout.to(DEV))
    assert _lib.device_status() == 0
    # the bound of the other oracle tests of these kernels: four roundings of the element type; fp32: sums of 256 products
    bound = {torch.bfloat16: 4 * 2.0 ** -9, torch.float16: 4 * 2.0 ** -12, torch.float32: 4e-6}[dtype]
    for got, ref in zip([out] + [x.grad for x in leaves], [want] + [x.grad for x in want_in]):
        got, ref = got.detach().float().cpu(), ref.detach().float()
        assert torch.isfinite(got).all()
        assert (got - ref).norm() <= bound * ref.norm()
