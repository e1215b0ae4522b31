"""Head counts that leave the last group of query heads partly filled (five heads of a tensor-parallel shard, say), with
batches whose shares go from such a group to the next sequence's full one after items of several tiles: the warps of the
heads that were not there then join in the middle of the tile rings.  CPU: that the batches hold such shares.  GPU:
every kernel shape on them against the oracle."""
import pytest
import torch

from tests.helpers import assert_close, oracle_for
from wsvd_b200 import _lib, inputs, ops
from wsvd_b200.kernel.flash_decoding import (
    token_decode_attention_flash_int8_latent_per_head_decoding_rope as op_i8,
    token_decode_attention_flash_latent_per_head_decoding_rope as op_f16,
)

SMS = 148
# dtype, heads, lengths, rank, rows of the cache
CASES = [
    (torch.int8, 5, [8192] * 16, 64, "head"),
    (torch.int8, 6, [1024] * 64, 64, "head"),
    (torch.int8, 7, [2048 - 100 * i for i in range(17)] * 2, 48, "head"),
    (torch.int8, 5, [1536, 900, 2048, 1024] * 10, 64, "scattered"),
    (torch.int8, 6, [1024] * 64, 64, "pages of 16"),
    (torch.int8, 5, [2048] * 40, 62, "head"),
    (torch.int8, 6, [1024, 700] * 32, 62, "scattered"),
    (torch.float16, 7, [2048] * 32, 64, "head"),
    (torch.float16, 5, [1024, 1500] * 30, 64, "scattered"),
    (torch.float16, 3, [2048] * 50, 64, "pages of 16"),
    (torch.float16, 5, [2048] * 40, 62, "head"),
]


def _rejoins(lens, heads, group):
    """Per CTA of a balanced launch: tiles of the items that only part of the group's heads have, where the CTA goes on
    with an item that more of them have."""
    lib = _lib.lib()
    n_hg = -(-heads // group)
    items = [(min(group, heads - hg * group), t) for n in lens for hg in range(n_hg) for t in range(-(-n // 128))]
    total = len(items)
    found = []
    for c in range(min(SMS, total)):
        mine = items[lib.wsvd_share_begin(c, total, SMS):lib.wsvd_share_begin(c + 1, total, SMS)]
        run = []  # [heads, tiles] of the CTA's items
        for i, (g, t) in enumerate(mine):
            if i == 0 or t == 0:
                run.append([g, 0])
            run[-1][1] += 1
        found += [a[1] for a, b in zip(run, run[1:]) if b[0] > a[0]]
    return found


@pytest.mark.parametrize("dtype,heads,lens,rank,rows", CASES)
def test_the_batches_hold_such_shares(dtype, heads, lens, rank, rows):
    found = _rejoins(lens, heads, 2 if dtype == torch.float16 else 4)
    assert len(found) >= 8 and max(found) >= 3, found


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,heads,lens,rank,rows", CASES)
def test_against_the_oracle(dtype, heads, lens, rank, rows):
    base = inputs.make_case(len(lens), heads, 128, rank, rank, lens, max(lens), seed=heads + rank, latent_dtype=dtype)
    case = base if rows == "head" else inputs.token_major_copy(base, shuffle_seed=5, page_size=16 if "16" in rows else 1)
    c = case.to("cuda")

    def run():
        if dtype == torch.int8:
            return op_i8(c.q, c.infer_state, heads, 128, c.latent_k, c.k_scale, c.latent_v, c.v_scale, c.wk, None)
        return op_f16(c.q, c.infer_state, heads, 128, c.latent_k, c.latent_v, c.wk)

    got = run()
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    assert_close(got, oracle_for(base), f"{dtype} {heads} heads {rows}")
    for _ in range(5):
        assert torch.equal(run(), got), "bitwise repeatable"
