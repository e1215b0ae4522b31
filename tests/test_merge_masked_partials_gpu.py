"""Partials without any weight (log-sum-exp -inf, the way a block is masked out) in the merges, wherever they stand among
the batches of eight that the merges take at a time."""
import pytest
import torch

from tests.helpers import assert_close, oracle_for
from wsvd_b200 import inputs, ops
from wsvd_b200.kernel.flash_decoding import token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8

pytestmark = pytest.mark.gpu
INF = float("inf")


@pytest.mark.parametrize("n", [1, 8, 9, 17, 40])
@pytest.mark.parametrize("where", ["front", "middle", "back", "all but the first", "all but the last", "all", "none"])
def test_merge_kernel(n, where):
    g = torch.Generator().manual_seed(n)
    B, H, W, S = 2, 3, 64, 128
    mid = torch.randn(B, H, n, W, generator=g)
    lse = torch.randn(B, H, n, generator=g)
    third = max(1, n // 3)
    masked = {"front": range(min(n - 1, max(third, 8))), "middle": range(third, min(n - 1, 2 * third)),
              "back": range(max(1, n - third), n), "all but the first": range(1, n),
              "all but the last": range(n - 1), "all": range(n), "none": range(0)}[where]
    lse[1, 1, list(masked)] = -INF
    want = (torch.softmax(lse.double(), -1)[..., None] * mid.double()).sum(2)  # (NaN where no partial has weight)
    out = torch.zeros(B, H, W, dtype=torch.float16, device="cuda")
    ops.decode_stage2(mid.cuda(), lse.cuda(), torch.full((B,), n * S, dtype=torch.int32, device="cuda"), out, S)
    torch.cuda.synchronize()
    if where == "all":
        assert torch.isnan(out[1, 1]).all()
        out[1, 1], want[1, 1] = 0, 0
    # fp32 sums of at most 40 terms and __expf (2 ulp): below 1e-5 of values of at most ~5; one f16 rounding (2^-11)
    assert_close(out, want, f"{n} {where}", atol=1e-5, rtol=6e-4)


def test_a_lost_value_of_a_masked_partial_stays_lost():
    """0 x NaN is a NaN, as in the sum that takes one partial after another."""
    mid, lse = torch.ones(1, 1, 9, 8), torch.zeros(1, 1, 9)
    lse[0, 0, :8] = -INF
    mid[0, 0, 2, 5] = float("nan")
    out = torch.zeros(1, 1, 8, dtype=torch.float16, device="cuda")
    ops.decode_stage2(mid.cuda(), lse.cuda(), torch.tensor([9 * 32], dtype=torch.int32, device="cuda"), out, 32)
    torch.cuda.synchronize()
    assert torch.isnan(out[0, 0, 5]) and (out[0, 0, [0, 1, 2, 3, 4, 6, 7]] == 1).all()


@pytest.mark.parametrize("masked_tiles", [1, 8, 9, 20])
def test_merge_inside_the_kernel(masked_tiles):
    """One sequence over many CTAs, of which the first ones see scores of -inf alone: positive products of q and K (q on
    the slowest pair of frequencies alone, positive factors and latents) under a scale of -inf."""
    n, H, cut = 8192, 8, masked_tiles * 128
    case = inputs.make_case(1, H, 128, 64, 64, [n], n, seed=3)
    case.q.zero_()
    case.q[..., 63] = 1.0
    case.wk.copy_(case.wk.abs().clamp(min=0.05))
    case.wk.view(64, H, 128)[..., 127] = 0.0  # the rotation by less than pi / 2 keeps the product positive
    st = case.storage["latent_k"]
    st.copy_((st.int().abs() + 1).clamp(max=127).to(torch.int8))
    want = oracle_for(case)
    c = case.to("cuda")
    run = lambda: op_i8(c.q, c.infer_state, H, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None)
    whole = run()
    assert_close(whole, want, "nothing masked")
    slots = c.infer_state.req_manager.req_to_token_indexs[0, :cut].long()
    c.k_scale[slots] = -INF
    got = run()
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    # the same with a finite score far below all others, whose weight is zero in fp32 too
    c.k_scale[slots] = -60000.0
    low = run()
    torch.cuda.synchronize()
    assert torch.isfinite(got).all() and not torch.equal(got, whole)
    assert_close(got, low.float().cpu(), f"{masked_tiles} tiles masked", atol=1e-5, rtol=6e-4)


def test_partials_of_the_lowest_finite_weight_count():
    lowest = -torch.finfo(torch.float32).max
    mid, lse = torch.arange(9.0).view(1, 1, 9, 1).expand(1, 1, 9, 8).contiguous(), torch.full((1, 1, 9), -INF)
    lse[0, 0, [2, 8]] = lowest
    out = torch.zeros(1, 1, 8, dtype=torch.float16, device="cuda")
    ops.decode_stage2(mid.cuda(), lse.cuda(), torch.tensor([9 * 32], dtype=torch.int32, device="cuda"), out, 32)
    torch.cuda.synchronize()
    assert (out == 5).all()  # (2 + 8) / 2
