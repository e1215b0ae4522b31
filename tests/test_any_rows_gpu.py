"""Ranks and row addresses that the tensor copies cannot take, by AUTO, against the oracle: even ones on the tcgen05
kernel, odd ones on the generic kernel."""
import pytest
import torch

from oracle import latent_decode_oracle as orc
from tests.helpers import assert_close, oracle_for
from wsvd_b200 import inputs, ops
from wsvd_b200.kernel.flash_decoding import (
    token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8,
    token_decode_attention_flash_latent_per_head_decoding_rope as op_f16,
)

pytestmark = pytest.mark.gpu
LENS = [2047, 1, 0, 1300, 129, 2048]


def _op(c, wv=False, kernel="auto"):
    H = c.q.shape[1]
    kw = dict(wv=c.wv if wv else None, kernel=kernel)
    if c.latent_k.dtype == torch.int8:
        out = op_i8(c.q, c.infer_state, H, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None, **kw)
    else:
        out = op_f16(c.q, c.infer_state, H, 128, c.latent_k, c.latent_v, c.wk, **kw)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    return out


@pytest.mark.parametrize("dtype,rk,rv", [
    (torch.int8, 62, 62), (torch.int8, 63, 61), (torch.int8, 1, 50), (torch.int8, 64, 47), (torch.int8, 17, 64),
    (torch.float16, 62, 62), (torch.float16, 2, 64), (torch.float16, 64, 54), (torch.float16, 50, 6)])
@pytest.mark.parametrize("heads", [5, 8])
def test_ranks(dtype, rk, rv, heads):
    case = inputs.make_case(len(LENS), heads, 128, rk, rv, LENS, max(LENS), seed=rk + heads, latent_dtype=dtype)
    c = case.to("cuda")
    lat, out = _op(c), _op(c, wv=True)
    assert_close(lat, oracle_for(case), f"{dtype} rank {rk}/{rv}")
    assert_close(out, oracle_for(case, wv=True), f"{dtype} rank {rk}/{rv} with U_v")
    assert (lat[2] == 0).all()
    assert torch.equal(lat, _op(c)), "bitwise repeatable"


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16])
@pytest.mark.parametrize("shift", [1, 4, 7, 8, 15])
@pytest.mark.parametrize("pitch", [0, 1, 6])
def test_row_addresses(dtype, shift, pitch):
    """Caches that start `shift` elements into their allocation, with token rows `pitch` elements longer than the heads
    need: rows at even alignments within 16 bytes (the others go to the generic kernel), token-major and scattered over the slots."""
    base = inputs.make_case(6, 6, 128, 64, 48, LENS, max(LENS), seed=shift, latent_dtype=dtype)
    case = inputs.token_major_copy(base, shuffle_seed=3)
    c = case.to("cuda")

    def move(x):
        T, H, R = x.shape
        buf = torch.zeros(shift + T * (H * R + pitch), dtype=x.dtype, device="cuda")
        view = buf.as_strided((T, H, R), (H * R + pitch, R, 1), shift)
        view.copy_(x)
        return view

    c.latent_k, c.latent_v = move(c.latent_k), move(c.latent_v)
    assert_close(_op(c), oracle_for(base), f"shift {shift} pitch {pitch}")


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16])
def test_grouped_query_heads_rank_62(dtype):
    base = inputs.make_case(6, 3, 128, 62, 62, LENS, max(LENS), seed=2, latent_dtype=dtype)
    q = torch.randn(6, 12, 128, generator=torch.Generator().manual_seed(1)).half()
    c = base.to("cuda")
    c.q = q.cuda()
    s = base.infer_state
    want, _ = orc.latent_decode_oracle(q, s.b_seq_len, s.b_req_idx, s.req_manager.req_to_token_indexs, base.latent_k,
                                       base.k_scale, base.latent_v, base.v_scale, base.wk)
    assert_close(_op(c), want, "gqa 4")


def test_rank_62_gather_over_ranks_takes_the_merge_kernel_when_rows_are_not_16_bytes():
    """O_lat rows of 62 values: no 16-byte peer stores, so the separate merge kernel delivers them."""
    from wsvd_b200 import _lib

    case = inputs.make_case(6, 6, 128, 62, 62, LENS, max(LENS), seed=5)
    c = case.to("cuda")
    out = torch.zeros(6, 6, 64, dtype=torch.float16, device="cuda")
    flags = torch.full((8,), 5, dtype=torch.int32, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    ps = _lib.PeerSet()
    ps.out[0], ps.flags[0], ps.counter = out.data_ptr(), flags.data_ptr(), counter.data_ptr()
    ps.n_peers, ps.rank, ps.head_offset, ps.epoch = 1, 0, 0, 5
    ps.out_stride_b, ps.out_stride_h, ps.timeout_ms = out.stride(0), out.stride(1), 1000
    ops.latent_decode_gather(c.q, c.infer_state, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None, ps)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    assert_close(out[:, :, :62], oracle_for(case), "gathered O_lat")
    assert (out[:, :, 62:] == 0).all()
