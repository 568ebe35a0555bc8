"""The fp32 kernels on 64 x 64 tiles against float64, at sizes where a tile can go wrong."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("be,qb,kb,tk", [(64, 1, 1, 1), (64, 3, 9, 7), (128, 2, 5, 3), (256, 1, 4, 4)])
def test_fp32_tiles_match_float64(be, qb, kb, tk, D, monkeypatch):
    from simple_vsa_b200 import b200_sparse_attention
    g = torch.Generator().manual_seed(be + kb + D)
    B, H = 1, 2
    q, dout = (torch.randn(B, H, qb * be, D, generator=g) for _ in range(2))
    k, v = (torch.randn(B, H, kb * be, D, generator=g) for _ in range(2))
    sizes = torch.tensor(([be, 1, 0, 63, 64, 65 % be + 1, be - 1] * 2)[:kb])
    for x in (k, v):       # whatever lies in the padding rows must not reach a result
        x.view(B, H, kb, be, D)[:, :, torch.arange(be)[None, :] >= sizes[:, None]] = float("nan")
    clean = [torch.nan_to_num(x, nan=0.0) for x in (k, v)]
    selected = torch.rand(B, H, qb, kb, generator=g)
    selected[..., 0] = 2.0                                # block 0 is full: every row has a live key
    selected = selected.topk(tk, dim=-1).indices.to(torch.int32)

    want_in = [x.double().requires_grad_() for x in (q, *clean)]
    rows = []
    for h in range(H):
        for i in range(qb):
            sel = selected[0, h, i].long()
            kk, vv = (x[0, h].view(kb, be, D)[sel].reshape(-1, D) for x in want_in[1:])
            live = (torch.arange(be)[None, :] < sizes[sel][:, None]).reshape(-1)
            s = (want_in[0][0, h, i * be:(i + 1) * be] @ kk.T) * D ** -0.5
            rows.append(s.masked_fill(~live, -torch.inf).softmax(-1) @ vv)
    want = torch.stack(rows).view(1, H, qb * be, D)
    want.backward(dout.double())

    def run(mode):
        monkeypatch.setenv("VSA_B200_KERNELS", mode)
        leaves = [x.to(DEV).requires_grad_() for x in (q, k, v)]
        out = b200_sparse_attention(*leaves, selected.to(DEV), sizes, block_size=(1, 1, be))
        out.backward(dout.to(DEV))
        return [out.detach()] + [x.grad for x in leaves]

    tiles, rows_kernel = run(""), run("scalar")
    for got, old, ref in zip(tiles, rows_kernel, [want] + [x.grad for x in want_in]):
        ref = ref.detach()
        error = [(x.cpu().double() - ref).norm() / ref.norm() for x in (got, old)]
        # sums of up to 1024 products of 2^-24 roundings each; and no further from float64 than the row kernels, whose own
        # error moves by a quarter with the order of the sums
        assert error[0] <= 2e-6
        assert error[0] <= 1.25 * error[1] + 1e-7


@pytest.mark.parametrize("be,D", [(64, 64), (128, 128), (256, 64)])
def test_padded_key_rows_get_exactly_zero_gradients_beside_a_nan(be, D):
    """A query row whose gradient holds NaN or infinity poisons the live rows of the key blocks that it reads, as in every
    kernel; their padding rows stay at zero."""
    from simple_vsa_b200 import b200_sparse_attention
    g = torch.Generator().manual_seed(be)
    nb, sizes = 4, torch.tensor([be, 5, be - 1, be // 2])
    q, k, v, dout = (torch.randn(1, 1, nb * be, D, generator=g).to(DEV) for _ in range(4))
    dout[0, 0, 3, 1], dout[0, 0, be + 2, 0] = float("nan"), float("inf")
    selected = torch.arange(nb, dtype=torch.int32).expand(1, 1, nb, nb).contiguous().to(DEV)
    leaves = [x.requires_grad_() for x in (q, k, v)]
    b200_sparse_attention(*leaves, selected, sizes, block_size=(1, 1, be)).backward(dout)
    dead = (torch.arange(be)[None, :] >= sizes[:, None]).view(-1).to(DEV)
    for x in leaves[1:]:
        assert torch.isnan(x.grad[0, 0, ~dead]).any()
        assert (x.grad[0, 0, dead] == 0).all()
