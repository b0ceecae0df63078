"""Short batches, where a unit of the persistent kernel is one tile whose KV blocks its two softmax groups take in
turn: lists of no, one, two, an odd and an even number of blocks, more units than SMs, every mask form."""
import pytest
import torch

from conftest import assert_parity
from omni_attention_b200 import create_causal_omni_block_mask, omni_attention, omni_attention_forward_out
from omni_attention_b200.inputs import random_fcp_block_mask
from oracle import omni_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("softcap", [None, 4.0])
@pytest.mark.parametrize("block", [128, 64])
@pytest.mark.parametrize("D,dtype", [(32, torch.float16), (64, torch.bfloat16), (128, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("H,nq,rest", [(1, 1, 0), (2, 2, 5), (3, 5, 63), (1, 9, 1), (38, 8, 0)])
def test_lists_of_any_length(cuda_device, H, nq, rest, D, dtype, block, softcap):
    """Against the oracle with the tolerance of the parity contract. 38 heads of 8 tiles are just past the rule
    and run as pairs (split units that outnumber the SMs: test_long_lists_in_both_block_sizes). `rest` tokens are missing from the last block."""
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


@pytest.mark.parametrize("H", [2, 150])   # 150 heads of two tiles are more pairs than SMs: the pair form
@pytest.mark.parametrize("D,dtype", [(32, torch.float16), (64, torch.bfloat16), (128, torch.bfloat16)])
def test_rows_that_are_zero_whatever_the_inputs_hold(cuda_device, H, D, dtype):
    """Rows beyond the sequence, rows without a key and rows with NaN scores are zero with log-sum-exp -inf in both
    forms, also where q, k or v is not finite; every other row has the bits of the call on finite inputs."""
    g = torch.Generator().manual_seed(D)
    n, padded = 200, 256
    q, k, v = (torch.randn(1, H, padded, D, generator=g).to(dtype).to(cuda_device) for _ in range(3))
    bm = create_causal_omni_block_mask(1, H, n, n)
    # the diagonal tile of the second Q block element by element, row 170 without any key there ...
    tile = torch.ones(128, 128, dtype=torch.bool).tril()
    tile[170 - 128] = False
    bm.block_mask_types[:, :, 1, 1] = 3
    bm.partial_block_mask_indices = torch.full_like(bm.kv_indices, -1)
    bm.partial_block_mask_indices[:, :, 1, 1] = 0
    bm.partial_block_masks = tile[None]
    # ... and only that tile listed, so that row 170 attends nothing
    bm.kv_num_blocks[:, :, 1] = 1
    bm.kv_indices[:, :, 1, 0], bm.block_mask_types[:, :, 1, 0], bm.partial_block_mask_indices[:, :, 1, 0] = 1, 3, 0

    def call(q, v):
        out, lse = torch.full_like(q, 7.0), torch.zeros(1, H, padded, device=cuda_device)
        omni_attention_forward_out(q, k, v, out, bm, n, lse=lse)
        return out, lse

    want, want_lse = call(q, v)
    bad_q, bad_v = q.clone(), v.clone()
    bad_q[:, :, n:] = float("nan")
    bad_q[:, :, n + 3] = float("inf")
    bad_q[:, :, 77, 3] = float("nan")
    bad_v[:, :, 199, 5] = float("inf")   # key 199 is seen by row 199 alone, but its block is visited by all of the tile
    out, lse = call(bad_q, bad_v)
    zero = torch.zeros(padded, dtype=torch.bool, device=cuda_device)
    zero[n:] = zero[77] = zero[170] = True
    assert bool((out[:, :, zero] == 0).all()) and bool((lse[:, :, zero] == -float("inf")).all())
    rest = ~zero
    assert torch.equal(lse[:, :, rest], want_lse[:, :, rest])
    first = rest.clone()
    first[128:] = False
    assert torch.equal(out[:, :, first], want[:, :, first])
    cols = [c for c in range(D) if c != 5]   # 0 * Inf in column 5 of the rows that visit the block
    assert torch.equal(out[:, :, rest][..., cols], want[:, :, rest][..., cols])


@pytest.mark.parametrize("H,nq", [(1, 240), (1, 296), (1, 297), (2, 148), (3, 100)])
def test_long_lists_in_both_block_sizes(cuda_device, H, nq):
    """Few heads of long sequences, up to and past the most tiles that take the split form: the same mask in 64- and in
    128-blocks has the same bits at head_dim 128, where the tables of 64-blocks are what fills shared memory."""
    n = nq * 128 - 70
    g = torch.Generator(device=cuda_device).manual_seed(nq)
    q, k, v = (torch.randn(1, H, n, 128, generator=g, device=cuda_device).mul_(0.5).bfloat16() for _ in range(3))
    masks = [create_causal_omni_block_mask(1, H, n, n, block, block, cuda_device) for block in (128, 64)]
    (a, la), (b, lb) = (omni_attention(q, k, v, m, return_lse=True) for m in masks)
    assert torch.equal(a, b) and torch.equal(la, lb)
    rows = torch.tensor([0, 1, 127, 128, n // 2, n - 1], device=cuda_device)   # a few rows in fp32
    s = q[:, :, rows].float() @ k.float().transpose(-1, -2) / 128 ** 0.5
    s = s.masked_fill(torch.arange(n, device=cuda_device) > rows[:, None], float("-inf"))
    assert_parity(a[:, :, rows], la[:, :, rows], s.softmax(-1) @ v.float(), s.logsumexp(-1), f"{H} x {nq}")
