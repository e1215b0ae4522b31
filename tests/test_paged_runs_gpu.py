"""Tiles made of several runs of token slots: pages smaller than the 128-token tile, and a prompt in one
run followed by scattered slots."""
import pytest
import torch

from tests.helpers import assert_close, oracle_for
from wsvd_b200 import inputs, ops
from wsvd_b200.infer_state import InferState
from wsvd_b200.kernel.flash_decoding import token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8

pytestmark = pytest.mark.gpu


def _run(case, heads):
    c = case.to("cuda")
    got = op_i8(c.q, c.infer_state, heads, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None, kernel="tc")
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    return got


@pytest.mark.parametrize("page_size", [8, 16, 32])
@pytest.mark.parametrize("rk,rv", [(64, 48), (32, 64)])
def test_small_pages(page_size, rk, rv):
    base = inputs.make_case(4, 6, 128, rk, rv, [1025, 301, 1792, 17], 1792, seed=page_size)
    got = _run(inputs.token_major_copy(base, shuffle_seed=4, page_size=page_size), 6)
    assert_close(got, oracle_for(base), f"page_size={page_size}")


@pytest.mark.parametrize("tail", [1, 40, 200])
def test_prompt_run_then_scattered_slots(tail):
    """The last `tail` tokens of every sequence sit in slots of their own, in no order."""
    lens = [700, 333, 1280]
    base = inputs.make_case(3, 6, 128, 64, 64, lens, 1280, seed=tail)
    plain = inputs.token_major_copy(base)
    s = plain.infer_state
    table = s.req_manager.req_to_token_indexs.clone()
    T = plain.latent_k.shape[0]
    extra = T + torch.randperm(3 * tail, generator=torch.Generator().manual_seed(1)).to(torch.int32)

    def grow(x):
        return torch.cat([x, torch.zeros((3 * tail,) + tuple(x.shape[1:]), dtype=x.dtype)])

    for name in ("latent_k", "latent_v", "k_scale", "v_scale"):
        x = grow(getattr(plain, name))
        for b, n in enumerate(lens):
            x[extra[b * tail:(b + 1) * tail].long()] = x[table[b, n - tail:n].long()]
        setattr(plain, name, x)
    for b, n in enumerate(lens):
        table[b, n - tail:n] = extra[b * tail:(b + 1) * tail]
    plain.infer_state = InferState(3, 1280, lens, device="cpu", req_to_token=table)
    assert_close(_run(plain, 6), oracle_for(base), f"tail={tail}")
