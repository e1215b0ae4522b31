"""int8 caches whose rows the tensor copies cannot take (rank 62): scales of either sign, zeros and NaNs, as the warp-MMA
kernel and the oracle have them."""
import pytest
import torch

from tests.helpers import assert_close, oracle_for
from wsvd_b200 import inputs, ops
from wsvd_b200.kernel.flash_decoding import token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8

pytestmark = pytest.mark.gpu
LENS = [2047, 1, 0, 1300, 129, 2048]
NAN = float("nan")


def _case(heads=8):
    return inputs.make_case(len(LENS), heads, 128, 62, 62, LENS, max(LENS), seed=heads)


def _run(c, kernel="auto", **kw):
    out = op_i8(c.q, c.infer_state, c.q.shape[1], 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None, kernel=kernel, **kw)
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    return out


@pytest.mark.parametrize("share", [0.01, 0.5, 1.0])
@pytest.mark.parametrize("layout", ["head", "scattered"])
def test_negative_and_zero_scales(share, layout):
    case = _case(7)
    g = torch.Generator().manual_seed(1)
    for name in ("k_scale", "v_scale"):
        sc = case.storage[name]
        sign = torch.where(torch.rand(sc.shape, generator=g) < share, -1.0, 1.0)
        sign[torch.rand(sc.shape, generator=g) < 0.02] = 0.0
        sc.copy_((sc.float() * sign).half())
    lv = case.storage["latent_v"]
    lv[torch.rand(lv.shape, generator=g) < 0.05] = -128  # the one value without a negative
    want = oracle_for(case)
    if layout == "scattered":
        case = inputs.token_major_copy(case, shuffle_seed=3)
    c = case.to("cuda")
    got = _run(c)
    assert_close(got, want, f"{share} of the scales negative")
    assert torch.equal(got, _run(c)), "bitwise repeatable"


@pytest.mark.parametrize("what", ["v_scale", "k_scale", "q"])
def test_nans_make_their_row_nan(what):
    """One NaN in the middle of a sequence, one in a sequence of a single token, one head whose every score is a NaN."""
    c = _case().to("cuda")
    slots = c.infer_state.req_manager.req_to_token_indexs
    good = _run(c)
    if what == "q":
        c.q[0, 3, 5] = c.q[1, 2, 0] = NAN
        rows = [(0, 3), (1, 2)]
    else:
        sc = getattr(c, what)
        sc[slots[0, 777].long(), 3] = NAN
        sc[slots[1, 0].long(), 2] = NAN
        sc[slots[4, :129].long(), 1] = NAN
        rows = [(0, 3), (1, 2), (4, 1)]
    got, mma = _run(c), _run(c, "mma")
    bad = torch.zeros(good.shape, dtype=torch.bool, device="cuda")
    for b, h in rows:
        bad[b, h] = True
    assert torch.equal(torch.isnan(got), bad) and torch.equal(torch.isnan(mma), bad)
    assert torch.equal(got[~bad], good[~bad])
