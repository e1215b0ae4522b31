"""f16 latents on the tcgen05 kernel (batches of at least one 128-token tile per SM) against the oracle."""
import pytest
import torch

from oracle import latent_decode_oracle as orc
from tests.helpers import assert_close, oracle_for
from wsvd_b200 import inputs, ops
from wsvd_b200.kernel.flash_decoding import token_decode_attention_flash_latent_per_head_decoding_rope as op_f16

pytestmark = pytest.mark.gpu
LENS = [2047, 1, 0, 1300, 129, 2048]


def _case(heads=7, rk=64, rv=64, lens=LENS, seed=3):
    return inputs.make_case(len(lens), heads, 128, rk, rv, lens, max(lens), seed=seed, latent_dtype=torch.float16)


def _run(case, kernel="auto", wv=False, **kw):
    c = case.to("cuda")
    out = op_f16(c.q, c.infer_state, c.q.shape[1], 128, c.latent_k, c.latent_v, c.wk, wv=c.wv if wv else None,
                 kernel=kernel, **kw)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    return out


@pytest.mark.parametrize("rk,rv", [(64, 64), (64, 48), (8, 64), (40, 16)])
@pytest.mark.parametrize("heads", [2, 7])
def test_ranks_ragged_lengths_poisoned_padding(rk, rv, heads):
    """Padding holds NaN; one sequence is empty, one has a single token; the last group of two heads holds one."""
    lens = LENS * (4 if heads == 2 else 1)
    case = _case(heads, rk, rv, lens)
    lat, out = _run(case), _run(case, wv=True)
    assert_close(lat, oracle_for(case), f"rank {rk}/{rv}")
    assert_close(out, oracle_for(case, wv=True), f"rank {rk}/{rv} with U_v")
    assert (lat[2] == 0).all() and (out[2] == 0).all()
    assert torch.equal(lat, _run(case)), "bitwise repeatable"
    # another kernel ran than the warp-MMA one (their sums differ in the last bit somewhere)
    assert not torch.equal(lat, _run(case, "mma"))


@pytest.mark.parametrize("page_size", [1, 16, 64, 128])
def test_paged_cache(page_size):
    base = _case(6, lens=[1025, 300, 1792, 17, 2048, 640])
    case = inputs.token_major_copy(base, shuffle_seed=4, page_size=page_size)
    assert_close(_run(case), oracle_for(base), f"page_size={page_size}")


def test_interleaved_pairing_and_position_offsets():
    case = _case(8)
    assert_close(_run(case, rope_layout="interleaved"), oracle_for(case, rope_layout="interleaved"), "interleaved")
    off = torch.tensor([5, 0, 77, 1000, 3, 250], dtype=torch.int32)
    assert_close(_run(case, pos_offset=off.cuda()), oracle_for(case, pos_offset=off), "pos_offset")


@pytest.mark.parametrize("gqa", [2, 3, 4])
@pytest.mark.parametrize("scattered", [False, True])
def test_grouped_query_heads(gqa, scattered):
    hkv = 3
    base = _case(hkv, seed=gqa)
    q = torch.randn(len(LENS), hkv * gqa, 128, generator=torch.Generator().manual_seed(gqa)).half()
    case = inputs.token_major_copy(base, shuffle_seed=2) if scattered else base
    c = case.to("cuda")
    got = op_f16(q.cuda(), c.infer_state, hkv * gqa, 128, c.latent_k, c.latent_v, c.wk)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    s = base.infer_state
    want, _ = orc.latent_decode_oracle(q, s.b_seq_len, s.b_req_idx, s.req_manager.req_to_token_indexs, base.latent_k, None,
                                       base.latent_v, None, base.wk)
    assert_close(got, want, f"gqa {gqa}")


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nan_and_infinities_reach_the_output(bad):
    """A NaN in q or K makes the head's row NaN; an infinite value latent of a token with weight makes its rank infinite."""
    case = _case(8)
    c = case.to("cuda")
    s = c.infer_state
    run = lambda q=c.q, lk=c.latent_k, lv=c.latent_v: op_f16(q, s, 8, 128, lk, lv, c.wk)
    good = run()
    q = c.q.clone()
    q[3, 1, 5] = bad
    got = run(q=q)
    assert torch.isnan(got[3, 1]).all() and torch.equal(got[3, 2:], good[3, 2:]) and torch.equal(got[0], good[0])
    slot = int(s.req_manager.req_to_token_indexs[3, 40])
    keep = c.latent_v[slot, 2, 7].clone()
    c.latent_v[slot, 2, 7] = bad
    got = run()
    c.latent_v[slot, 2, 7] = keep
    assert not torch.isfinite(got[3, 2, 7]) and torch.isnan(got[3, 2, 7]) == (bad != bad)
    assert torch.isfinite(got[3, 2, :7]).all() and torch.equal(got[3, 1], good[3, 1])


def test_one_dominant_token_and_peaked_weights():
    """Scores over a wide range: references of the value sums that move often, weights far below the largest."""
    case = _case(4, lens=[2048, 2000, 1999, 2048, 1500, 1024, 900, 800], seed=11)
    case.q.mul_(12.0)
    # Against the warp-MMA kernel, whose score operands are rounded to f16 in the same way: that rounding moves a
    # score by up to |score| 2^-10 or so, with q twelve times as large as the op's tolerance is meant for.  What is
    # left is the order of fp32 sums in the scores (|z| up to ~60: 60 * 2^-23 * 128 terms < 1e-3 in the exponent)
    # and one f16 rounding of each output.
    assert_close(_run(case), _run(case, "mma").cpu(), "peaked", atol=1e-3, rtol=2e-3)
    case.q.mul_(0.0)
    assert_close(_run(case), oracle_for(case, dtype=torch.float64), "flat")


def test_partials_entry_then_merge_kernel():
    """Stage 1 alone with the balanced shares, merged by the separate kernel (unaligned output of a gather)."""
    import ctypes as ct

    from wsvd_b200 import _lib

    case = _case(6)
    c = case.to("cuda")
    s = c.infer_state
    out = torch.zeros(6, 6, 130, dtype=torch.float16, device="cuda")[:, :, 1:129]  # rows at odd offsets: no 16-byte stores
    ps = _lib.PeerSet()
    flags = torch.full((8,), 5, dtype=torch.int32, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    ps.out[0], ps.flags[0], ps.counter = out.data_ptr(), flags.data_ptr(), counter.data_ptr()
    ps.n_peers, ps.rank, ps.head_offset, ps.epoch = 1, 0, 0, 5
    ps.out_stride_b, ps.out_stride_h, ps.timeout_ms = out.stride(0), out.stride(1), 1000
    ops.latent_decode_gather(c.q, s, c.latent_k, None, c.latent_v, None, c.wk, None, ps, wv=c.wv)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    assert_close(out, oracle_for(case, wv=True), "merge kernel after balanced f16 shares")
