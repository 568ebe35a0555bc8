"""The operator in one native call per direction against the separate entry points, which the timing hook still uses; and
the one-CTA route inversion at the edges of its range."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,be,D,gated", [(torch.bfloat16, 64, 128, True), (torch.float16, 128, 64, False),
                                              (torch.float32, 64, 64, True), (torch.float32, 4, 8, False)])
def test_one_call_equals_the_separate_entry_points(dtype, be, D, gated, monkeypatch):
    from simple_vsa_b200 import _lib, video_sparse_attn
    g = torch.Generator().manual_seed(3)
    B, H, Qb, Kb, tk = 2, 3, 5, 11, 4
    q, dout, gate = (torch.randn(B, H, Qb * be, D, generator=g).to(dtype).to(DEV) for _ in range(3))
    k, v = (torch.randn(B, H, Kb * be, D, generator=g).to(dtype).to(DEV) for _ in range(2))
    kv_sizes, q_sizes = torch.full((Kb,), be), torch.full((Qb,), be)
    kv_sizes[3], q_sizes[1] = be // 2, be - 1

    def run():
        leaves = [x.clone().requires_grad_() for x in ((q, k, v, gate) if gated else (q, k, v))]
        out, aux = video_sparse_attn(*leaves[:3], kv_sizes, q_sizes, tk, (1, 1, be), leaves[3] if gated else None, return_aux=True)
        return [out.detach(), aux["coarse_scores"], aux["selected"]] + list(torch.autograd.grad(out, leaves, dout))

    one = run()
    calls = []
    monkeypatch.setattr(_lib, "recorder", lambda name, what, stream: calls.append(name))
    many = run()
    assert "vsa_topk" in calls and "vsa_sparse_bwd_dkdv_fused" in calls and "vsa_operator_fwd" not in calls
    for i, (a, b) in enumerate(zip(one, many)):
        if i in (4, 5):      # dK and dV: the in-edges of a key block come in no fixed order, an fp32 sum's last bits with them
            unit = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]
            assert (a - b).abs().max().float() <= 2 * unit * b.abs().max().float()
        else:
            assert torch.equal(a, b)
