"""The tensor-core kernels on blocks of 128 and 256 tokens (128-row tcgen05 kernels, and those that take their place on small
grids and short routes; head dims 64 and 128) at the edges of their tiles, against the CPU oracle: live sizes around 0, 1, 64,
128 and the full block, a single tile, odd tile counts, more tiles than any ring is deep, query and key lengths that differ."""

import pytest
import torch

from oracle import vsa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("be,qb,kb,tk", [(128, 1, 1, 1), (128, 2, 5, 4), (128, 3, 7, 5), (256, 2, 5, 3), (256, 1, 9, 9)])
@pytest.mark.parametrize("large", [False, True])
def test_blocks_of_128_rows_match_the_oracle(be, qb, kb, tk, D, dtype, large):
    from simple_vsa_b200 import _lib, b200_sparse_attention
    g = torch.Generator().manual_seed(be + 7 * kb + D)
    # a few row tiles take the 64-row kernels; one full wave of 128-row tiles takes the others (head dim 64, short routes: mma.sync)
    B, H = 1, 296 // (qb * be // 64) if large else 2
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    for p, n in enumerate((qb, qb, kb)):
        kernels = 3 if large else 2
        if D == 64 and p < 2 and tk * be // 64 < (8, 4)[p]:
            kernels = 1
        if large and D == 128 and p == 0 and tk * be // 64 <= 16:
            kernels = 2
        assert _lib.lib.vsa_sparse_pass_kernels(p, B * H, n * be, D, be, tk, code) == kernels
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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("be,qb", [(128, 400), (256, 200)])
def test_dq_of_query_blocks_without_a_live_key_is_the_pooled_gradient_alone(be, qb, D, dtype):
    """Every other query block routes to empty blocks only, or outside the key table only: nothing of its own Q may reach its
    dQ, which is the pooled gradient's share (or zero without one), and the blocks between them are what they are beside
    ordinary neighbours."""
    from simple_vsa_b200 import _lib
    g = torch.Generator().manual_seed(be + D)
    BH, Kb, tk, scale = 2, 8, 5, D ** -0.5
    Lq, Lkv, code = qb * be, Kb * be, _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    new = lambda *shape: torch.randn(*shape, generator=g).to(dtype).to(DEV)
    q, dout, k, v, dq_mean = new(BH, Lq, D), new(BH, Lq, D), new(BH, Lkv, D), new(BH, Lkv, D), new(BH, qb, D)
    kv_sizes = torch.tensor([be, be // 2 + 3, 1, 0, 0, be, 0, 65], dtype=torch.int32, device=DEV)
    q_sizes = torch.randint(0, be + 1, (qb,), generator=g, dtype=torch.int32)
    ordinary = torch.rand(BH, qb, Kb, generator=g)
    ordinary[..., 5] = 2.0                                # a full block in every row
    ordinary = ordinary.topk(tk, dim=-1).indices.to(torch.int32)
    dead = torch.arange(qb) % 2 == 1
    routes = ordinary.clone()
    routes[:, dead] = torch.tensor([3, 4, 6, -2, 3], dtype=torch.int32)
    routes[:, torch.arange(qb) % 4 == 3] = torch.tensor([-1, Kb, 2 ** 30, Kb + 1, -8], dtype=torch.int32)
    st = torch.cuda.current_stream().cuda_stream

    def run(table, pooled):
        sel, qs = table.to(DEV), q_sizes.to(DEV)
        out, dq = torch.empty_like(q), torch.full_like(q, float("nan"))
        lse, delta = torch.empty(BH, Lq, device=DEV), torch.empty(BH, Lq, device=DEV)
        _lib.call("vsa_sparse_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), sel.data_ptr(), kv_sizes.data_ptr(), out.data_ptr(),
                  lse.data_ptr(), BH, Lq, Lkv, D, be, tk, scale, code, st)
        args = [dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), sel.data_ptr(),
                kv_sizes.data_ptr(), delta.data_ptr(), dq.data_ptr()] + ([dq_mean.data_ptr(), qs.data_ptr()] if pooled else [])
        _lib.call("vsa_sparse_bwd_dq" + ("_fused" if pooled else ""), *args, BH, Lq, Lkv, D, be, tk, scale, code, st)
        torch.cuda.synchronize()
        return out.cpu().view(BH, qb, be, D), dq.cpu().view(BH, qb, be, D)

    rows = torch.arange(be)[None, :, None] < q_sizes[:, None, None]
    share = torch.where(rows, dq_mean.cpu().float()[:, :, None] / q_sizes.clamp(min=1)[:, None, None], torch.zeros(())).to(dtype)
    for pooled, want in ((False, torch.zeros_like(share)), (True, share)):
        (out, dq), (out_ref, dq_ref) = run(routes, pooled), run(ordinary, pooled)
        assert torch.equal(dq[:, dead], want[:, dead])
        assert torch.isnan(out[:, dead].float()).all()
        assert torch.equal(dq[:, ~dead], dq_ref[:, ~dead]) and torch.equal(out[:, ~dead], out_ref[:, ~dead])
    assert _lib.device_status() == 0


def test_small_fp16_probabilities_at_head_dim_64_are_as_precise_as_on_the_warp_level_kernels(monkeypatch):
    """One key 12 nats above 5000 others: their probabilities sit near the bottom of fp16, and the output is made of them."""
    from simple_vsa_b200 import _lib, ops
    g = torch.Generator().manual_seed(12)
    be, qb, kb, D, H = 128, 2, 40, 64, 64
    q, k, v = (torch.randn(1, 1, n * be, D, generator=g) for n in (qb, kb, kb))
    k *= 0.5
    v += 1.0
    q[..., 0], k[..., 0] = 4.0, 0.0
    k[0, 0, 5], v[0, 0, 5] = 0.0, 0.0
    k[0, 0, 5, 0] = 12.0 * D ** 0.5 / 4.0
    q, k, v = (x.half() for x in (q, k, v))
    assert _lib.lib.vsa_sparse_pass_kernels(0, H, qb * be, D, be, kb, _lib.VSA_F16) == 3        # H equal heads
    want = (q[0, 0].double() @ k[0, 0].double().T * D ** -0.5).softmax(-1) @ v[0, 0].double()
    q, k, v = (x.expand(1, H, -1, D).contiguous() for x in (q, k, v))
    selected = torch.arange(kb, dtype=torch.int32).expand(1, H, qb, kb).contiguous().to(DEV)
    sizes = torch.full((kb,), be, dtype=torch.int32, device=DEV)
    error = {}
    for mode in ("auto", "mma"):
        monkeypatch.setenv("VSA_B200_KERNELS", mode)
        out, lse = ops.sparse_forward(q.to(DEV), k.to(DEV), v.to(DEV), selected, sizes, be, D ** -0.5, True)
        error[mode] = (out[0, 0].double().cpu() - want).norm() / want.norm()
    # the same probabilities rounded at the same binades; what differs is the order of the fp32 sums around them
    assert error["auto"] <= 1.05 * error["mma"]


@pytest.mark.parametrize("dtype,k_factor,q_factor", [(torch.bfloat16, 8.0, 40.0), (torch.float16, 1.5, 20.0)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("be,qb", [(128, 2), (256, 1)])
def test_one_half_of_a_tile_outside_the_shift_range_is_recomputed_exactly(be, qb, D, dtype, k_factor, q_factor):
    """The softmax shift of a row comes from its first live key tile, here one of 5 keys.  A later block scores hundreds of binades
    above it for the rows 64 to 127 of a tile (out of the element type's range: the exact kernel's work) and a few for the rows
    before them.  Output, statistic and combined output match the oracle in both halves."""
    from simple_vsa_b200 import _lib, ops
    g = torch.Generator().manual_seed(be + D)
    # routes long enough for the 128-row forward; blocks 8 and up are empty
    H, (kb, tk), scale = 296 // (qb * be // 64), (8, 6) if be == 256 else (12, 10), D ** -0.5
    q, gate = (torch.randn(1, H, qb * be, D, generator=g) for _ in range(2))
    k, v = (torch.randn(1, H, kb * be, D, generator=g) for _ in range(2))
    out_c = torch.randn(1, H, qb, D, generator=g).to(dtype)
    q.view(1, H, -1, 128, D)[:, :, :, 64:] *= q_factor
    k.view(1, H, kb, be, D)[:, :, 3] *= k_factor
    q, k, v, gate = (x.to(dtype) for x in (q, k, v, gate))
    sizes = torch.tensor([5, be, be, be - 3, be, 64, be, 1] + [0] * (kb - 8))
    selected = torch.rand(1, H, qb, kb, generator=g)
    selected[..., 0], selected[..., 3] = 3.0, 2.0           # the block of 5 keys comes first, the high-scoring one second
    selected = selected.topk(tk, dim=-1).indices.to(torch.int32)
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    assert _lib.lib.vsa_sparse_pass_kernels(0, H, qb * be, D, be, tk, code) == 3
    # the scores say which rows leave the range: 2^(score - shift) in fp32, fp16's 2^16 and bf16's 2^127 above it
    s = torch.einsum("bhtd,bhsd->bhts", q.float(), k.float().view(1, H, kb, be, D)[:, :, [0, 3]].flatten(2, 3)) * scale * 1.4427
    above = (s[..., be:2 * be - 3].amax(-1) - s[..., :5].amax(-1)).view(1, H, -1, 128)
    limit = 127 if dtype == torch.bfloat16 else 16
    assert (above[..., 64:].amax(-1) > limit + 10).all() and (above[..., :64] < limit - 2).all()
    want, want_lse = O.sparse_attention(q, k, v, selected, sizes, be, return_lse2=True)
    want_total = O.combine(want.to(dtype), out_c, gate, be, dtype)
    out, lse, total = ops.sparse_forward(q.to(DEV), k.to(DEV), v.to(DEV), selected.to(DEV), sizes.to(DEV, torch.int32), be, scale,
                                         True, combine_with=(out_c.to(DEV), gate.to(DEV)))
    assert _lib.device_status() == 0
    for got, ref, rtol in ((out, want, 2e-2), (total, want_total, 2e-2), (lse, want_lse, 1e-3)):
        torch.testing.assert_close(got.float().cpu(), ref.float(), atol=2e-2 if rtol == 2e-2 else 5e-2, rtol=rtol)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("live", [1, 2, 3, 4, 7])
def test_the_128_row_forward_on_routes_with_few_live_tiles(live, D, dtype):
    """Long routes of mostly empty blocks: one to seven live tiles, fewer than its softmax groups or its rings hold and more, and
    query blocks without any."""
    from simple_vsa_b200 import _lib, ops
    g = torch.Generator().manual_seed(live + D)
    be, qb, kb, tk, H, scale = 128, 2, 10, 9, 74, D ** -0.5
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    assert _lib.lib.vsa_sparse_pass_kernels(0, H, qb * be, D, be, tk, code) == 3
    q = torch.randn(1, H, qb * be, D, generator=g).to(dtype)
    k, v = (torch.randn(1, H, kb * be, D, generator=g).to(dtype) for _ in range(2))
    sizes = torch.tensor(([be, 1, 63, 64, 65, be, 127])[:live] + [0] * (kb - live))
    for x in (k, v):                                      # whatever lies in the padding rows must not reach a result
        x.view(1, H, kb, be, D)[:, :, torch.arange(be)[None, :] >= sizes[:, None]] = float("nan")
    clean = [torch.nan_to_num(x.float(), nan=0.0).to(dtype) for x in (k, v)]
    selected = torch.rand(1, H, qb, kb, generator=g)
    selected[..., 0] = 2.0                                # block 0 is full: every row has a live key ...
    selected = selected.topk(tk, dim=-1).indices.to(torch.int32)
    selected[:, ::2, 1] = kb - 1                          # ... but in these query blocks none has
    want, want_lse = O.sparse_attention(q, *clean, selected, sizes, be, return_lse2=True)
    out, lse = ops.sparse_forward(q.to(DEV), k.to(DEV), v.to(DEV), selected.to(DEV), sizes.to(DEV, torch.int32), be, scale, True)[:2]
    assert _lib.device_status() == 0
    out, lse = out.float().cpu().view(1, H, qb, be, D), lse.cpu().view(1, H, qb, be)
    dead = torch.zeros(1, H, qb, dtype=torch.bool)
    dead[:, ::2, 1] = True
    assert torch.isnan(out[dead]).all()
    want, want_lse = want.float().view_as(out)[~dead], want_lse.float().view_as(lse)[~dead]
    bound = 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12)         # as above
    assert (out[~dead] - want).norm() <= bound * want.norm()
    # a score is a sum of D <= 128 products in fp32: off by at most 128 * 2^-24 * sum |q k| * scale * log2 e, sum |q k| below 300
    assert (lse[~dead] - want_lse).abs().max() <= 1e-3
