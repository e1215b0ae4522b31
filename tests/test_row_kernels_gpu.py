"""The element-wise row kernels at the edges of their vector path, against the torch chains they replace."""
import pytest
import torch

from wsvd_b200 import ops

pytestmark = pytest.mark.gpu


def _norm(x):
    xf = x.float()
    return (xf * torch.rsqrt(xf.pow(2).mean(dim=-1, keepdim=True) + 1e-5)).half()


# 8: one vector; 2048: one per thread; 2056: a second pass of one vector; 16384: the widest row in registers; 16392: past
# it; 100 and 4097: no whole vectors
@pytest.mark.parametrize("cols", [8, 100, 2048, 2056, 4096, 4097, 16384, 16392])
@pytest.mark.parametrize("rows", [1, 5])
@pytest.mark.parametrize("shift", [0, 1])
def test_rms_norm_and_residual(cols, rows, shift):
    g = torch.Generator().manual_seed(cols)
    n = rows * cols

    def make(scale):  # shift: the matrix starts 2 bytes into its allocation, so no 16-byte vectors
        buf = torch.empty(n + shift, dtype=torch.float16, device="cuda")
        buf[shift:] = (torch.randn(n, generator=g) * scale).half().cuda()
        return buf[shift:].view(rows, cols)

    x, d = make(1.0), make(0.7)
    # one f16 rounding of the result: half a unit in the last place of f16, and the fp32 sum's order
    tol = dict(rtol=1.1e-3, atol=1e-6)
    torch.testing.assert_close(ops.rms_norm(x), _norm(x), **tol)
    s, y = ops.add_rms_norm(x, d)
    assert torch.equal(s, x + d)
    torch.testing.assert_close(y, _norm(x + d), **tol)
    # the vector and the scalar kernel add the squares in the same order: the same bits at any alignment
    other = torch.empty(n + 1, dtype=torch.float16, device="cuda")[1 - shift:n + 1 - shift].view(rows, cols)
    other.copy_(x)
    assert torch.equal(ops.rms_norm(other), ops.rms_norm(x))
    assert torch.equal(ops.add_rms_norm(other, d)[1], y)


@pytest.mark.parametrize("cols,ld,shift", [(8, 16, 0), (11008, 22016, 0), (1000, 2004, 0), (30, 64, 0), (64, 136, 1)])
def test_silu_mul(cols, ld, shift):
    g = torch.Generator().manual_seed(cols)
    buf = torch.randn(7 * ld + 8, generator=g).half().cuda()
    m = buf[shift:shift + 7 * ld].view(7, ld)
    up, gate = m[:, :cols], m[:, ld - cols:]
    want = up * torch.nn.functional.silu(gate.float()).half()
    # two f16 roundings (the silu, the product)
    torch.testing.assert_close(ops.silu_mul(up, gate), want, rtol=2e-3, atol=1e-6)
