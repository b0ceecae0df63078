"""Short batches, where a unit of the persistent kernel is one tile whose KV blocks its two softmax groups take in
turn: lists of no, one, two, an odd and an even number of blocks, more units than SMs, every mask form."""
import pytest
import torch

from conftest import assert_parity
from omni_attention_b200 import omni_attention
from omni_attention_b200.inputs import random_fcp_block_mask
from oracle import omni_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("softcap", [None, 4.0])
@pytest.mark.parametrize("block", [128, 64])
@pytest.mark.parametrize("D,dtype", [(32, torch.float16), (64, torch.bfloat16), (128, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("H,nq,rest", [(1, 1, 0), (2, 2, 5), (3, 5, 63), (1, 9, 1), (38, 8, 0)])
def test_lists_of_any_length(cuda_device, H, nq, rest, D, dtype, block, softcap):
    """Against the oracle with the tolerance of the parity contract. 38 heads of 8 tiles are 304 units, two or
    three for each SM. `rest` tokens are missing from the last block."""
    g = torch.Generator().manual_seed(100 * nq + D)
    padded = nq * 128
    bm = random_fcp_block_mask(1, H, padded, seed=nq, block=block)
    per = 128 // block
    if nq > 2:   # one tile without any work, and one whose first list is cut to a single block
        bm.kv_num_blocks[:, :, per:2 * per] = 0
        bm.kv_num_blocks[:, :, 2 * per] = 1
    n = padded - rest
    q, k, v = (torch.randn(1, H, n, D, generator=g).to(dtype) for _ in range(3))
    out, lse = omni_attention(*(t.to(cuda_device) for t in (q, k, v)), bm, return_lse=True, softcap=softcap)
    heads = sorted({0, H - 1})
    ro, rl = orc.block_mask_attention(q, k, v, bm, bh=[(0, h) for h in heads], softcap=softcap)
    for h in heads:
        live = torch.isfinite(rl[0, h])
        got_o, got_l = out[0, h].cpu(), lse[0, h].cpu()
        assert bool((got_o[~live] == 0).all()) and bool((got_l[~live] == -float("inf")).all())
        assert_parity(got_o[live], got_l[live], ro[0, h][live], rl[0, h][live], f"head {h}")
    again = omni_attention(*(t.to(cuda_device) for t in (q, k, v)), bm, softcap=softcap)
    assert torch.equal(out, again)
