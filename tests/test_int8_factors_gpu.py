"""int8 U_k with column scales on the tcgen05 kernel: the vector build of its query-side operand and the
byte-wise one (rows that are not 8-byte aligned) against the oracle."""
import pytest
import torch

from oracle import latent_decode_oracle as orc
from tests.helpers import assert_close
from wsvd_b200 import inputs, ops
from wsvd_b200.kernel.flash_decoding import token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rope_layout", ["half", "interleaved"])
@pytest.mark.parametrize("rk", [16, 48, 64])
@pytest.mark.parametrize("pad", [0, 8, 3])
def test_int8_wk(rope_layout, rk, pad):
    """pad: columns in front of and behind the factor in memory (8: still 8-byte rows, 3: byte-wise)."""
    case = inputs.make_case(2, 6, 128, rk, 64, [300, 129], 304, seed=rk + pad)
    w8, sc = orc.quantize_per_token(case.wk.t().contiguous())  # one scale per output column
    wide = torch.zeros(rk, w8.shape[0] + 2 * pad, dtype=torch.int8)
    wide[:, pad:pad + w8.shape[0]] = w8.t()
    c = case.to("cuda")
    wk, ws = wide.cuda()[:, pad:pad + w8.shape[0]], sc.reshape(-1).cuda()
    got = op_i8(c.q, c.infer_state, 6, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, wk, ws, kernel="tc",
                rope_layout=rope_layout)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    s = case.infer_state
    want, _ = orc.latent_decode_oracle(case.q, s.b_seq_len, s.b_req_idx, s.req_manager.req_to_token_indexs, case.latent_k,
                                       case.k_scale, case.latent_v, case.v_scale, w8.t().contiguous(), sc.reshape(1, -1),
                                       rope_layout=rope_layout)
    assert_close(got, want, f"int8 wk rank {rk} {rope_layout} pad {pad}")
