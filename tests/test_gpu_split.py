"""The 64-row tcgen05 kernels that put a tile of the other side on each lane half (blocks of 64 tokens at head dims 64 and 128, larger
blocks on small grids; at head dim 64 the shortest routes run on mma.sync, as each test says) at the edges of their tiles, against
the CPU oracle: odd and single tile counts (one half without a tile), more pairs than any ring is deep, live sizes around 0, 1, 32
(a part of V) and the full tile, query and key lengths that differ, whatever bits the padding rows hold, and score gaps beyond the
range of the softmax shift."""

import pytest
import torch

from oracle import vsa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("be,qb,kb,tk", [(64, 1, 1, 1), (64, 3, 2, 2), (64, 5, 9, 3), (64, 4, 23, 17), (64, 26, 21, 8), (256, 1, 3, 1)])
def test_64_row_tiles_match_the_oracle(be, qb, kb, tk, D, dtype):
    from simple_vsa_b200 import _lib, b200_sparse_attention
    g = torch.Generator().manual_seed(be + 7 * kb + D)
    B, H = 1, 3
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    if be == 64 or D == 128:                              # head dim 64: short routes run on mma.sync
        for p, n in enumerate((qb, qb, kb)):
            assert _lib.lib.vsa_sparse_pass_kernels(p, B * H, n * be, D, be, tk, code) == (1 if D == 64 and tk < (8, 4, 2)[p] else 2)
    q, dout = (torch.randn(B, H, qb * be, D, generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, H, kb * be, D, generator=g).to(dtype) for _ in range(2))
    sizes = torch.tensor(([be, 1, 0, 32, be - 1, 33, be, 31, be] * 3)[:kb])
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
    # operands, P and dS carry 2^-9 (bf16) or 2^-12 (fp16) each, summed over many keys: relative 2-norm error near one rounding,
    # far below four of them
    bound = 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    for got, ref in zip([out] + [x.grad for x in leaves], [want] + [x.grad for x in want_in]):
        got, ref = got.detach().float().cpu(), ref.detach().float()
        assert torch.isfinite(got).all()
        assert (got - ref).norm() <= bound * ref.norm()
    dead = torch.arange(be)[None, :] >= sizes[:, None]
    for x in leaves[1:]:
        assert (x.grad.view(B, H, kb, be, D)[:, :, dead.to(DEV)] == 0).all()


@pytest.mark.parametrize("dtype,k_factor", [(torch.bfloat16, 8.0), (torch.float16, 1.5)])
@pytest.mark.parametrize("D", [64, 128])
def test_a_tile_outside_the_shift_range_is_recomputed_exactly(D, dtype, k_factor):
    """A block later in the route scores hundreds of binades above the first pair for every other query block."""
    from simple_vsa_b200 import _lib, ops
    g = torch.Generator().manual_seed(D)
    be, H, qb, kb, tk, scale = 64, 2, 6, 9, 7, D ** -0.5
    q = torch.randn(1, H, qb * be, D, generator=g)
    k, v = (torch.randn(1, H, kb * be, D, generator=g) for _ in range(2))
    q.view(1, H, qb, be, D)[:, :, 1::2] *= 40.0 if dtype == torch.bfloat16 else 20.0
    k.view(1, H, kb, be, D)[:, :, 3] *= k_factor
    q, k, v = (x.to(dtype) for x in (q, k, v))
    sizes = torch.tensor([5, 9, be, be, be - 3, be, 64, be, 1])
    selected = torch.tensor([0, 1, 2, 3, 4, 5, 8], dtype=torch.int32).expand(1, H, qb, tk).contiguous()
    want, want_lse = O.sparse_attention(q, k, v, selected, sizes, be, return_lse2=True)
    out, lse = ops.sparse_forward(q.to(DEV), k.to(DEV), v.to(DEV), selected.to(DEV), sizes.to(DEV, torch.int32), be, scale, True)[:2]
    assert _lib.device_status() == 0
    torch.testing.assert_close(out.float().cpu(), want.float(), atol=2e-2, rtol=2e-2)
    torch.testing.assert_close(lse.float().cpu(), want_lse.float(), atol=5e-2, rtol=1e-3)


@pytest.mark.parametrize("D,tk", [(128, 40), (64, 40)])
def test_many_ragged_tiles_leave_their_neighbours_alone(D, tk, monkeypatch):
    """Half the blocks ragged, two CTAs on every SM, twenty pairs each: clearing the padding rows of one pair must not reach the rows
    of the pair before it, whatever the timing.  Against the warp-level kernels: two roundings of values around 1 in bf16 apart."""
    from simple_vsa_b200 import _lib, ops
    g = torch.Generator(device=DEV).manual_seed(D)
    be, H, nb = 64, 8, 200
    q, k, v = (torch.randn(1, H, nb * be, D, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    sizes = torch.randint(1, 2 * be, (nb,), device=DEV, generator=g, dtype=torch.int32).clamp(max=be)
    selected = torch.rand(1, H, nb, nb, device=DEV, generator=g).topk(tk, dim=-1).indices.to(torch.int32)
    outs = {}
    for mode in ("auto", "mma"):
        monkeypatch.setenv("VSA_B200_KERNELS", mode)
        outs[mode] = [ops.sparse_forward(q, k, v, selected, sizes, be, D ** -0.5, True)[0] for _ in range(5)]
    assert _lib.device_status() == 0
    want = outs["mma"][0].float()
    for out in outs["auto"]:
        assert torch.equal(out, outs["auto"][0])
        # P carries 2^-9 and the output 2^-9 of values below 1/2: a cleared row of V would show as one of ~1500 weights, times |v|
        assert (out.float() - want).abs().max() < 4e-3


@pytest.mark.parametrize("qb", [1, 2, 3])
@pytest.mark.parametrize("D", [64, 128])
def test_a_key_that_nobody_attends_to_keeps_finite_gradients(D, qb):
    """A key whose score is -inf for every query has probability zero: its dK and dV are exactly zero, as they are in the formula,
    also where an odd number of query tiles leaves half of the last pair without a tile (zero rows times an infinite key are NaN)."""
    from simple_vsa_b200 import _lib, b200_sparse_attention
    g = torch.Generator().manual_seed(qb + D)
    be, B, H, kb, tk = 64, 1, 2, 3, 2
    q, dout = (torch.randn(B, H, qb * be, D, generator=g).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, H, kb * be, D, generator=g).to(torch.bfloat16) for _ in range(2))
    q[..., 0] = q[..., 0].abs() + 0.5
    k[:, :, [3, 40], 0] = float("-inf")
    sizes = torch.tensor([be, 50, be])
    selected = torch.tensor([0, 1], dtype=torch.int32).expand(B, H, qb, tk).contiguous()
    want_in = [x.clone().requires_grad_() for x in (q, k, v)]
    want = O.sparse_attention(*want_in, selected, sizes, be)
    want.backward(dout.float())
    leaves = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    out = b200_sparse_attention(*leaves, selected.to(DEV), sizes, block_size=(1, 1, be))
    out.backward(dout.to(DEV))
    assert _lib.device_status() == 0
    bound = 4 * 2.0 ** -9                                  # as above
    for got, ref in ((out, want), (leaves[1].grad, want_in[1].grad), (leaves[2].grad, want_in[2].grad)):
        got, ref = got.detach().float().cpu(), ref.detach().float()
        assert torch.isfinite(ref).all() and torch.isfinite(got).all()
        assert (got - ref).norm() <= bound * ref.norm()
    for x in leaves[1:]:
        assert (x.grad[:, :, [3, 40]] == 0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("live", [1, 2, 3, 4, 7])
def test_routes_with_few_live_tiles(live, D, dtype):
    """Routes long enough for the 64-row kernels at either head dim, of mostly empty blocks: one live tile, one pair, an odd tail, and
    a query block without any; every key block is read by an odd number of query tiles."""
    from simple_vsa_b200 import _lib, b200_sparse_attention
    g = torch.Generator().manual_seed(live + D)
    be, B, H, qb, kb, tk = 64, 1, 2, 4, 9, 8
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    assert all(_lib.lib.vsa_sparse_pass_kernels(p, B * H, n * be, D, be, tk, code) == 2 for p, n in enumerate((qb, qb, kb)))
    q, dout = (torch.randn(B, H, qb * be, D, generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, H, kb * be, D, generator=g).to(dtype) for _ in range(2))
    sizes = torch.tensor(([be, 1, 32, 33, be, 31, be - 1])[:live] + [0] * (kb - live))
    for x in (k, v):
        x.view(B, H, kb, be, D)[:, :, torch.arange(be)[None, :] >= sizes[:, None]] = float("nan")
    clean = [torch.nan_to_num(x.float(), nan=0.0).to(dtype) for x in (k, v)]
    selected = torch.arange(tk, dtype=torch.int32).expand(B, H, qb, tk).contiguous()
    selected = selected[..., torch.randperm(tk, generator=g)].contiguous()
    selected[:, :, 2] = kb - 1                            # an empty block only
    rows = torch.arange(qb * be) // be != 2
    want_in = [q.clone().requires_grad_()] + [x.clone().requires_grad_() for x in clean]
    want = O.sparse_attention(want_in[0][:, :, rows], *want_in[1:], selected[:, :, [0, 1, 3]], sizes, be, q_blocks_per_chunk=8)
    want.backward(dout[:, :, rows].float())
    leaves = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    out = b200_sparse_attention(*leaves, selected.to(DEV), sizes, block_size=(1, 1, be))
    out.backward(dout.to(DEV))
    assert _lib.device_status() == 0
    assert torch.isnan(out[:, :, (~rows).to(DEV)].float()).all()
    assert (leaves[0].grad[:, :, (~rows).to(DEV)] == 0).all()
    bound = 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12)         # as above
    for got, ref in zip([out[:, :, rows.to(DEV)], leaves[0].grad[:, :, rows.to(DEV)]] + [x.grad for x in leaves[1:]],
                        [want, want_in[0].grad[:, :, rows]] + [x.grad for x in want_in[1:]]):
        got, ref = got.detach().float().cpu(), ref.detach().float()
        assert torch.isfinite(got).all()
        assert (got - ref).norm() <= bound * ref.norm()


@pytest.mark.parametrize("dtype,k_factor,q_factor", [(torch.bfloat16, 8.0, 40.0), (torch.float16, 1.5, 20.0)])
@pytest.mark.parametrize("D", [64, 128])
def test_a_recomputed_tile_takes_the_combine_with_it(D, dtype, k_factor, q_factor):
    """The rows that the exact kernel computes again reach the combined output too, gated, and their neighbours keep theirs."""
    from simple_vsa_b200 import _lib, ops
    g = torch.Generator().manual_seed(D)
    be, H, qb, kb, tk, scale = 64, 2, 6, 9, 8, D ** -0.5
    code = _lib.VSA_BF16 if dtype == torch.bfloat16 else _lib.VSA_F16
    assert _lib.lib.vsa_sparse_pass_kernels(0, H, qb * be, D, be, tk, code) == 2
    q, gate = (torch.randn(1, H, qb * be, D, generator=g) for _ in range(2))
    k, v = (torch.randn(1, H, kb * be, D, generator=g) for _ in range(2))
    out_c = torch.randn(1, H, qb, D, generator=g).to(dtype)
    q.view(1, H, qb, be, D)[:, :, 1::2] *= q_factor
    k.view(1, H, kb, be, D)[:, :, 3] *= k_factor
    q, k, v, gate = (x.to(dtype) for x in (q, k, v, gate))
    sizes = torch.tensor([5, 9, be, be, be - 3, be, 64, be, 1])
    selected = torch.tensor([0, 1, 2, 3, 4, 5, 6, 8], dtype=torch.int32).expand(1, H, qb, tk).contiguous()
    # the scores say which tiles leave the range: fp16 holds 2^16, bf16 2^127 above the shift (at head dim 128 fp16 is four binades above)
    s = torch.einsum("bhtd,bhsd->bhts", q.float(), k.float()) * scale * 1.4427
    s = s.view(1, H, qb, be, kb, be)
    first = torch.cat([s[:, :, :, :, 0, :5], s[:, :, :, :, 1, :9]], -1).amax(-1)
    above = (s[:, :, :, :, 3].amax(-1) - first).amax(-1)
    limit = 127 if dtype == torch.bfloat16 else 20
    assert (above[:, :, 1::2] > limit + 4).all() and (above[:, :, ::2] < (limit if dtype == torch.bfloat16 else 14)).all()
    want, want_lse = O.sparse_attention(q, k, v, selected, sizes, be, return_lse2=True)
    want_total = O.combine(want.to(dtype), out_c, gate, be, dtype)
    out, lse, total = ops.sparse_forward(q.to(DEV), k.to(DEV), v.to(DEV), selected.to(DEV), sizes.to(DEV, torch.int32), be, scale,
                                         True, combine_with=(out_c.to(DEV), gate.to(DEV)))
    assert _lib.device_status() == 0
    # the bounds of the test of the 128-row kernels' redo path
    for got, ref, rtol in ((out, want, 2e-2), (total, want_total, 2e-2), (lse, want_lse, 1e-3)):
        torch.testing.assert_close(got.float().cpu(), ref.float(), atol=2e-2 if rtol == 2e-2 else 5e-2, rtol=rtol)
