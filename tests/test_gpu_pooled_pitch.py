"""The pooled attention with padded rows of probabilities and dS: any block counts on the tensor cores."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Qb,Kb,D", [(1, 1, 128), (3, 7, 64), (8, 9, 128), (127, 129, 128), (130, 65, 64), (257, 1380, 128)])
def test_pooled_attention_with_padded_rows_matches_the_cuda_core_products(Qb, Kb, D, dtype, monkeypatch):
    from simple_vsa_b200 import _lib
    torch.manual_seed(Qb + Kb)
    BH, scale, pitch = 2, D ** -0.5, -(-Kb // 8) * 8
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    new = lambda *shape: torch.empty(*shape, device=DEV, dtype=dtype)
    qc, dco = (torch.randn(BH, Qb, D, device=DEV).to(dtype) for _ in range(2))
    kc, vc = (torch.randn(BH, Kb, D, device=DEV).to(dtype) for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream

    def run():
        scores, out_c = new(BH, Qb, Kb), new(BH, Qb, D)
        probs, ds = (torch.full((BH, Qb, pitch), float("nan"), device=DEV, dtype=dtype) for _ in range(2))
        rowdot = torch.empty(BH, Qb, device=DEV)
        dq, dk, dv = new(BH, Qb, D), new(BH, Kb, D), new(BH, Kb, D)
        _lib.call("vsa_coarse_fwd_pitched", qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), scores.data_ptr(), probs.data_ptr(),
                  out_c.data_ptr(), BH, Qb, Kb, pitch, D, scale, code, st)
        _lib.call("vsa_coarse_bwd_pitched", dco.data_ptr(), out_c.data_ptr(), qc.data_ptr(), kc.data_ptr(), vc.data_ptr(),
                  probs.data_ptr(), ds.data_ptr(), rowdot.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), BH, Qb, Kb,
                  pitch, D, scale, code, st)
        torch.cuda.synchronize()
        assert torch.isnan(probs[..., Kb:].float()).all() and torch.isnan(ds[..., Kb:].float()).all()    # never touched
        return scores, probs[..., :Kb], out_c, dq, dk, dv

    fast = run()
    monkeypatch.setenv("VSA_B200_KERNELS", "scalar")
    slow = run()
    assert _lib.device_status() == 0
    if Qb % 8 or Kb % 8:
        assert torch.equal(fast[0], slow[0])        # the scores, and with them the routes, are the same bits
    # the same roundings of the same 16-bit operands around fp32 sums in another order: half a unit flips now and then
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for a, b in zip(fast[1:], slow[1:]):
        a, b = a.float(), b.float()
        assert (a - b).abs().max() <= 2 * unit * b.abs().max() + 1e-6
        assert (a - b).norm() <= unit * b.norm() + 1e-6
