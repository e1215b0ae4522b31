"""When the layer leaves its element-wise chains to torch: wherever autograd follows one of its tensors."""
import pytest
import torch
from torch.autograd import forward_ad

from wsvd_b200 import layer_utils


def test_what_autograd_follows():
    x, w = torch.randn(2, 4), torch.randn(4, 4)
    assert not layer_utils._differentiated(x, w)
    w.requires_grad_()
    assert layer_utils._differentiated(x, w)
    with torch.no_grad():
        assert not layer_utils._differentiated(x, w)
    with forward_ad.dual_level():
        assert not layer_utils._differentiated(x)
        dual = forward_ad.make_dual(x, torch.ones_like(x))
        assert layer_utils._differentiated(dual, w)
        with torch.no_grad():  # forward mode goes on there
            assert layer_utils._differentiated(dual, w)
        assert not layer_utils._fused_rows(dual)


@pytest.mark.parametrize("device,dtype", [("cpu", torch.float32),
                                          pytest.param("cuda", torch.float16, marks=pytest.mark.gpu)])
def test_a_tangent_runs_through_the_chains(device, dtype):
    """The attention is opaque to autograd; the residual and the FFN are not."""
    g = torch.Generator().manual_seed(0)
    r = lambda *s: (torch.randn(*s, generator=g) * 0.5).to(device, dtype)
    D, H, R, M, F = 8, 2, 4, 16, 24
    w = dict(Wdq=r(M, H * R), Wdk=r(M, H * R), Wdv=r(M, H * R), Wuq=r(R, H * D), Wuvout=r(H, R, M), Wup=r(M, F),
             Wgate=r(M, F), Wdown=r(F, M))
    attn = lambda q: torch.zeros(q.shape[0], H, R, device=device, dtype=dtype)
    x, t = r(2, 1, M), r(2, 1, M)
    run = lambda x: layer_utils._layer(D, H, x, attn, **w)
    with forward_ad.dual_level():
        got = forward_ad.unpack_dual(run(forward_ad.make_dual(x, t))).tangent
    assert got is not None
    if dtype == torch.float32:
        step = 1e-3
        want = (run(x + step * t) - run(x - step * t)) / (2 * step)
    else:  # against the chain in fp32: a few f16 roundings (2^-11 each) of the values in between
        x, t, w = x.float(), t.float(), {k: v.float() for k, v in w.items()}
        attn = lambda q: torch.zeros(q.shape[0], H, R, device=device)
        with forward_ad.dual_level():
            want = forward_ad.unpack_dual(run(forward_ad.make_dual(x, t))).tangent
    # (central differences in fp32: 2^-24 / step = 6e-5 of values of a few tens)
    assert (got.float() - want).norm() <= 1e-2 * want.norm()
