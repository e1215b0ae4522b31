"""What WSVD_KERNEL_AUTO alone sends to the tcgen05 kernel (f16 latents, even ranks and rows that the tensor copies cannot
take), as far as the C ABI shows it without a GPU: what was refused stays refused, plans stay, workspaces never shrink."""
import ctypes

import pytest

from tests.test_cabi_cpu import _params
from wsvd_b200 import _lib

AUTO, GENERIC, TC, MMA = 0, 1, 2, 3
UNSUPPORTED = 7


def _p(rk, rv, dtype, kernel, **kw):
    f16 = dtype == 1
    args = dict(head_dim=128, rank_k=rk, rank_v=rv, latent_dtype=dtype, kernel=kernel, max_len=8192,
                k_scale=None if f16 else 0x1000, v_scale=None if f16 else 0x1000, k_stride_t=rk, k_stride_h=8192 * rk,
                v_stride_t=rv, v_stride_h=8192 * rv)
    args.update(kw)
    return _params(**args)


def _plan(p):
    sl, ns = ctypes.c_int32(), ctypes.c_int32()
    assert _lib.lib().wsvd_latent_decode_plan(ctypes.byref(p), ctypes.byref(sl), ctypes.byref(ns)) == 0
    return sl.value, ns.value


@pytest.mark.parametrize("rk,rv,dtype", [(64, 64, 1), (62, 62, 1), (62, 62, 0), (63, 64, 0), (64, 50, 0)])
def test_forced_tensor_core_kernel_still_refuses(rk, rv, dtype):
    p = _p(rk, rv, dtype, TC)
    need = _lib.lib().wsvd_latent_decode_workspace_bytes(ctypes.byref(p))
    assert _lib.lib().wsvd_latent_decode(ctypes.byref(p), ctypes.c_void_p(0x2000), need, None) == UNSUPPORTED


@pytest.mark.parametrize("rk,rv,dtype", [(64, 64, 1), (62, 62, 1), (62, 62, 0), (63, 64, 0), (16, 2, 1)])
@pytest.mark.parametrize("batch,max_len", [(1, 100), (2, 8192), (33, 3000), (300, 700)])
@pytest.mark.parametrize("split_len", [0, 256])
def test_plan_and_workspace_cover_the_kernel_it_ran_on_before(rk, rv, dtype, batch, max_len, split_len):
    auto = _p(rk, rv, dtype, AUTO, batch=batch, max_len=max_len, split_len=split_len)
    before = _p(rk, rv, dtype, MMA if rk % 2 == 0 else GENERIC, batch=batch, max_len=max_len, split_len=split_len)
    assert _plan(auto) == _plan(before)
    need = lambda p: _lib.lib().wsvd_latent_decode_workspace_bytes(ctypes.byref(p))
    assert need(auto) >= need(before)
    if split_len:  # fixed splits do not change kernels
        assert need(auto) == need(before)
