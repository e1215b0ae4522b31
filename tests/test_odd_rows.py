"""Odd ranks, odd strides and odd addresses under AUTO: the generic kernel, which computes in fp32 what the tensor-core
kernels round to f16, with its plan, its workspace and its room in the static entry."""
import ctypes

import pytest
import torch

from tests.helpers import assert_close, oracle_for
from tests.test_auto_routes_cpu import AUTO, GENERIC, _p, _plan
from wsvd_b200 import _lib, inputs, ops
from wsvd_b200.kernel.flash_decoding import (
    token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8,
    token_decode_attention_flash_latent_per_head_decoding_rope as op_f16,
)

I8, F16 = 0, 1
ROWS = [(I8, 63, 64, {}), (I8, 64, 61, {}), (I8, 64, 64, dict(k_stride_t=65)), (I8, 64, 64, dict(v_stride_h=8191)),
        (I8, 64, 64, dict(latent_k=0x1001)), (F16, 64, 64, dict(v_stride_t=65)), (F16, 62, 62, dict(latent_v=0x1002)),
        (F16, 63, 64, {})]


@pytest.mark.parametrize("dtype,rk,rv,kw", ROWS)
@pytest.mark.parametrize("batch,max_len", [(1, 100), (16, 8192), (300, 700)])
def test_plan_and_workspace_are_the_generic_kernels(dtype, rk, rv, kw, batch, max_len):
    auto = _p(rk, rv, dtype, AUTO, batch=batch, max_len=max_len, **kw)
    generic = _p(rk, rv, dtype, GENERIC, batch=batch, max_len=max_len, **kw)
    need = lambda p: _lib.lib().wsvd_latent_decode_workspace_bytes(ctypes.byref(p))
    assert _plan(auto) == _plan(generic) and need(auto) == need(generic)


def _odd(c, stride, shift):
    def move(x):
        T, H, R = x.shape
        buf = torch.zeros(shift + T * (H * R + stride), dtype=x.dtype, device="cuda")
        view = buf.as_strided((T, H, R), (H * R + stride, R, 1), shift)
        view.copy_(x)
        return view

    c.latent_k, c.latent_v = move(c.latent_k), move(c.latent_v)
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,rk,rv,stride,shift", [
    (torch.int8, 63, 61, 0, 0), (torch.int8, 64, 64, 1, 0), (torch.int8, 64, 48, 0, 1), (torch.float16, 64, 64, 1, 0),
    (torch.float16, 62, 62, 0, 1)])
def test_the_generic_kernels_bits(dtype, rk, rv, stride, shift):
    lens = [2048, 1300, 1, 0]
    base = inputs.make_case(4, 8, 128, rk, rv, lens, max(lens), seed=rk, latent_dtype=dtype)
    case = inputs.token_major_copy(base) if stride or shift else base
    c = case.to("cuda")
    if stride or shift:
        c = _odd(c, stride, shift)

    def run(kernel):
        if dtype == torch.int8:
            return op_i8(c.q, c.infer_state, 8, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None, kernel=kernel)
        return op_f16(c.q, c.infer_state, 8, 128, c.latent_k, c.latent_v, c.wk, kernel=kernel)

    got = run("auto")
    assert_close(got, oracle_for(base), f"{dtype} {rk}/{rv}")
    assert torch.equal(got, run("generic"))


@pytest.mark.gpu
@pytest.mark.parametrize("rank", [62, 63])
def test_static_entry_with_a_context_whose_table_would_not_fit(rank):
    """32768 positions make a table of 8 MB, all of the static scratch.  Rank 63 needs none; rank 62 is refused, as ever."""
    n = 32768
    case = inputs.make_case(1, 2, 128, rank, rank, [n], n, seed=rank)
    c = case.to("cuda")
    s = c.infer_state
    out = torch.empty(1, 2, rank, dtype=torch.float16, device="cuda")
    p, _keep = ops.build_params(c.q, s.b_seq_len, s.b_req_idx, s.req_manager.req_to_token_indexs, n, c.latent_k, c.k_scale,
                                c.latent_v, c.v_scale, c.wk, out=out)
    p.rope_table, p.rope_table_rows = None, 0
    status = _lib.lib().wsvd_latent_decode_static(ctypes.byref(p), None)
    if rank == 62:
        assert status == 8  # too large
        return
    assert status == 0
    torch.cuda.synchronize()
    assert_close(out, oracle_for(case), "odd rank, 32768 tokens, no table")
