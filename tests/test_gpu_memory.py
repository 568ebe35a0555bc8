"""Peak memory of the operator's backward: no pooled score matrix beside the gradients."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("be,L,D", [(64, 65536, 64), (4, 8192, 8)])     # the pooled dS fits into dQ; it is larger than dQ
def test_backward_holds_no_pooled_scores_beside_the_gradients(be, L, D):
    from simple_vsa_b200 import video_sparse_attn
    B, H, tk, dt = 1, 4, 2, torch.bfloat16
    nb = L // be
    sizes = torch.full((nb,), be, device=DEV, dtype=torch.int32)
    leaves = [torch.randn(B, H, L, D, device=DEV).to(dt).requires_grad_() for _ in range(3)]
    dout = torch.randn(B, H, L, D, device=DEV).to(dt)

    def peak_of_the_backward():
        out = video_sparse_attn(*leaves, sizes, sizes, tk, (1, 1, be))
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_stats()["requested_bytes.all.current"]
        torch.autograd.grad(out, leaves, dout)
        torch.cuda.synchronize()
        return torch.cuda.memory_stats()["requested_bytes.all.peak"] - before

    peak_of_the_backward()
    tensor, scores = B * H * L * D * 2, B * H * nb * nb * 2
    # pooled gradients (four tensors of nb rows), routes, statistics; every piece rounded up to 256 bytes
    small = B * H * (4 * nb * D * 2 + nb * (tk + 4) * 4 + L * 4) + 16 * 256
    assert small < scores                       # the bound below tells the two apart
    assert peak_of_the_backward() <= max(3 * tensor, scores) + small


def test_a_small_pooled_score_matrix_larger_than_dq_gives_the_same_gradients(monkeypatch):
    """64 blocks of 4 tokens at head dim 8: the pooled dS (64 columns a block row) does not fit into dQ (32) and sits in scratch."""
    from simple_vsa_b200 import _lib, video_sparse_attn
    torch.manual_seed(5)
    B, H, be, nb, D, tk = 1, 2, 4, 64, 8, 3
    sizes = torch.full((nb,), be, dtype=torch.int32)
    sizes[7] = 1
    leaves = [torch.randn(B, H, nb * be, D, device=DEV).requires_grad_() for _ in range(4)]
    dout = torch.randn(B, H, nb * be, D, device=DEV)

    def run():
        out = video_sparse_attn(*leaves[:3], sizes, sizes, tk, (1, 1, be), leaves[3])
        return torch.autograd.grad(out, leaves, dout)

    one = run()
    monkeypatch.setattr(_lib, "recorder", lambda name, what, stream: None)      # the separate entry points
    for a, b in zip(one, run()):
        # dK and dV sum their query rows in no fixed order: the last bits of sums of a few dozen products
        assert (a - b).abs().max() <= 2.0 ** -19 * b.abs().max()
