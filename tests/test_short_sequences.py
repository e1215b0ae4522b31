"""Short sequences under AUTO: what the tcgen05 kernel would run more slowly stays with the warp-MMA kernel, on either side of
each line of the rule."""
import ctypes

import pytest
import torch

from tests.helpers import assert_close, oracle_for
from tests.test_auto_routes_cpu import AUTO, MMA, _p
from wsvd_b200 import _lib, inputs
from wsvd_b200.kernel.flash_decoding import (
    token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8,
    token_decode_attention_flash_latent_per_head_decoding_rope as op_f16,
)

I8, F16 = 0, 1
# dtype, rank, batch, heads, longest sequence, whether it stays with the warp-MMA kernel
CASES = [
    (I8, 62, 40, 8, 32, True), (I8, 62, 40, 8, 33, False),
    (F16, 62, 40, 8, 255, True), (F16, 62, 40, 8, 256, False),
    (F16, 64, 40, 8, 96, True), (F16, 64, 40, 8, 97, False), (F16, 64, 40, 8, 128, False),
    (F16, 64, 40, 8, 129, True), (F16, 64, 40, 8, 160, True), (F16, 64, 40, 8, 161, False),
    (F16, 64, 148, 8, 160, True), (F16, 64, 149, 8, 160, False),
]


@pytest.mark.parametrize("dtype,rank,batch,heads,max_len,stays", CASES)
def test_workspace_shows_the_kernel(dtype, rank, batch, heads, max_len, stays):
    """The balanced mode's workspace holds prefix sums, arrival counters and a table of its own size on top."""
    need = lambda kernel: _lib.lib().wsvd_latent_decode_workspace_bytes(ctypes.byref(
        _p(rank, rank, dtype, kernel, batch=batch, n_q_heads=heads, n_kv_heads=heads, max_len=max_len)))
    assert need(AUTO) == need(MMA) if stays else need(AUTO) > need(MMA)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,rank,batch,heads,max_len,stays", [c for c in CASES if c[2] == 40])
def test_against_the_oracle(dtype, rank, batch, heads, max_len, stays):
    lens = [max_len] + [max(1, max_len - 3 * i) for i in range(1, batch)]
    case = inputs.make_case(batch, heads, 128, rank, rank, lens, max_len, seed=max_len,
                            latent_dtype=torch.int8 if dtype == I8 else torch.float16)
    c = case.to("cuda")

    def run(kernel):
        if dtype == I8:
            return op_i8(c.q, c.infer_state, heads, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None, kernel=kernel)
        return op_f16(c.q, c.infer_state, heads, 128, c.latent_k, c.latent_v, c.wk, kernel=kernel)

    got = run("auto")
    assert_close(got, oracle_for(case), f"{rank} {max_len}")
    assert torch.equal(got, run("mma")) == stays
