"""The operator on tensors whose length is no multiple of the block size, as they lie in memory, and the
one-kernel mask builder at the edges of its blocks."""
import pytest
import torch

from omni_attention_b200 import (block_mask_from_row_limits, create_omni_block_mask_from_modality_positions as build_mask,
                                 omni_attention, omni_attention_autograd, retile_block_mask)
from omni_attention_b200.ops import OmniAttnError, omni_attention_backward_out, omni_attention_forward_out

pytestmark = pytest.mark.gpu


def _limits(n, padded, g):
    """Row limits of a causal mask with one span attended in both directions."""
    lim = torch.arange(padded).clamp(max=n - 1)
    a = int(torch.randint(0, n, (1,), generator=g))
    b = min(n, a + int(torch.randint(1, 200, (1,), generator=g)))
    lim[a:b] = b - 1
    lim[n:] = n - 1
    return lim.view(1, padded)


@pytest.mark.parametrize("block", [128, 64])
@pytest.mark.parametrize("n", [1, 63, 65, 127, 129, 200, 383, 385])
@pytest.mark.parametrize("D,dtype", [(32, torch.float16), (64, torch.bfloat16), (128, torch.bfloat16)])
def test_unpadded_tensors_give_the_bits_of_padded_ones(cuda_device, n, D, dtype, block):
    """Forward, log-sum-exp and gradients of [1, 3, n, D] tensors against the same call on zero-padded
    copies through the padded entry points: the same tiles reach the tensor cores, so the bits are equal. Three
    heads back to back, so that reading past a head's end would read the next head."""
    g = torch.Generator().manual_seed(1000 * D + n)
    padded = -(-n // block) * block
    H = 3
    bm = block_mask_from_row_limits(_limits(n, padded, g), H, block=block)
    q, k, v, do = ((torch.randn(1, H, n, D, generator=g)).to(dtype).to(cuda_device) for _ in range(4))
    pad = lambda t, to: torch.nn.functional.pad(t, (0, 0, 0, to - n)).contiguous()
    out, lse = omni_attention(q, k, v, bm, return_lse=True)
    assert out.shape == q.shape and out.is_contiguous() and lse.shape == q.shape[:3]
    po, plse = torch.empty(1, H, padded, D, dtype=dtype, device=cuda_device), torch.empty(1, H, padded, device=cuda_device)
    omni_attention_forward_out(pad(q, padded), pad(k, padded), pad(v, padded), po, bm, n, lse=plse)
    assert torch.equal(out, po[:, :, :n]) and torch.equal(lse, plse[:, :, :n])

    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    got = torch.autograd.grad(omni_attention_autograd(*leaves, bm), leaves, do)
    bm128 = bm if block == 128 else retile_block_mask(bm, 128)
    p128 = bm128.q_len
    pq, pk, pv, pdo = (pad(t, p128) for t in (q, k, v, do))
    po, plse = torch.empty_like(pq), torch.empty(1, H, p128, device=cuda_device)
    omni_attention_forward_out(pq, pk, pv, po, bm128, n, lse=plse)
    want = [torch.empty_like(pq) for _ in range(3)]
    omni_attention_backward_out(pq, pk, pv, po, plse, pdo, *want, bm128, n)
    for a, b in zip(got, want):
        assert torch.equal(a, b[:, :, :n])


@pytest.mark.parametrize("n", [100, 128, 129, 512, 640, 1023, 1025, 2048])
def test_mask_builder_at_block_edges(cuda_device, n):
    """Spans that begin and end at, one before and one after block boundaries, overlap, are empty or reach past
    the end, for lengths with and without a rest: lists, types and tiles of the CPU builder."""
    spans = [[(0, 0, 1)], [(0, 127, 2)], [(0, 128, 128)], [(0, 129, 126)], [(0, 0, 128), (0, 128, 1)],
             [(0, 60, 300), (0, 100, 50), (0, 255, 2)], [(0, 5, 0), (0, n - 1, 1)], [(0, max(0, n - 130), 500)], [(0, 3, 4 * n)]]
    m = max(len(s) for s in spans)
    mp = torch.tensor([s + [(0, 0, 0)] * (m - len(s)) for s in spans], dtype=torch.int32)
    B, H = len(spans), 3
    cpu = build_mask(mp, B, H, n, n)
    gpu = build_mask(mp.to(cuda_device), B, H, n, n, device=cuda_device)
    for name in ("kv_num_blocks", "kv_indices", "block_mask_types"):
        assert torch.equal(getattr(gpu, name).cpu(), getattr(cpu, name)), name
    sel = cpu.partial_block_mask_indices >= 0
    gi = gpu.partial_block_mask_indices.cpu()
    assert torch.equal(gi >= 0, sel)
    assert gpu.partial_block_masks.shape == cpu.partial_block_masks.shape
    assert torch.equal(gpu.partial_block_masks.cpu()[gi[sel].long()],
                       cpu.partial_block_masks[cpu.partial_block_mask_indices[sel].long()])


@pytest.mark.parametrize("B,n,M", [(40, 8190, 8), (1300, 200, 2), (5000, 100, 3)])
def test_mask_builder_on_thousands_of_blocks(cuda_device, B, n, M):
    """Batches whose Q blocks are counted by kernels of their own (thousands of them, of 64, two and one for each batch
    element): lists, types, tiles and their order of the CPU builder."""
    g = torch.Generator().manual_seed(B)
    mp = torch.zeros(B, M, 3, dtype=torch.int32)
    mp[:, :, 1] = torch.randint(0, n + 50, (B, M), generator=g)
    mp[:, :, 2] = torch.randint(0, 400, (B, M), generator=g)
    cpu = build_mask(mp, B, 2, n, n)
    gpu = build_mask(mp.to(cuda_device), B, 2, n, n, device=cuda_device)
    for name in ("kv_num_blocks", "kv_indices", "block_mask_types"):
        assert torch.equal(getattr(gpu, name).cpu(), getattr(cpu, name)), name
    gi = gpu.partial_block_mask_indices.cpu()
    sel = gi[:, 0] >= 0
    assert torch.equal(gi >= 0, cpu.partial_block_mask_indices >= 0) and torch.equal(gi[:, 0], gi[:, 1])
    assert torch.equal(gi[:, 0][sel], torch.arange(int(sel.sum()), dtype=torch.int32))   # numbered in order, none twice
    assert gpu.partial_block_masks.shape == cpu.partial_block_masks.shape
    want = cpu.partial_block_masks[cpu.partial_block_mask_indices[:, 0][sel].long()]
    assert torch.equal(gpu.partial_block_masks[gi[:, 0][sel].long().to(cuda_device)].cpu(), want)


@pytest.mark.parametrize("n", [200, 383])
def test_views_that_start_at_any_element(cuda_device, n):
    """A length that is no multiple of the block may come as a view at any element offset (the rows are copied
    then, as padding copied them): outputs and gradients of the aligned copies."""
    g = torch.Generator().manual_seed(n)
    bm = block_mask_from_row_limits(_limits(n, -(-n // 128) * 128, g), 2)
    shape = (1, 2, n, 64)
    numel = 2 * n * 64
    view = lambda off: torch.randn(numel + 8, generator=g).half().to(cuda_device)[off:off + numel].view(shape)
    q, k, v, do = (view(off) for off in (1, 3, 4, 7))
    assert torch.equal(omni_attention(q, k, v, bm), omni_attention(q.clone(), k.clone(), v.clone(), bm))

    def grads(tensors, d_out):
        leaves = [t.detach().requires_grad_(True) for t in tensors]
        return torch.autograd.grad(omni_attention_autograd(*leaves, bm), leaves, d_out)

    for a, b in zip(grads((q, k, v), do), grads([t.clone() for t in (q, k, v)], do.clone())):
        assert torch.equal(a, b)


def test_a_call_waits_for_the_mask_and_not_for_later_work_of_its_stream(cuda_device):
    """A mask built on a side stream that goes on to other work: calls on another stream, and the first read of the byte
    pool, wait until the mask is there, but do not wait for that work."""
    n = 256
    mp = torch.tensor([[[0, 10, 50], [0, 100, 90]]], dtype=torch.int32, device=cuda_device)
    q = torch.randn(1, 2, n, 64, device=cuda_device).half()
    first = build_mask(mp, 1, 2, n, n, device=cuda_device)
    want, pool = omni_attention(q, q, q, first), first.partial_block_masks
    forward = torch.empty_like(q)
    omni_attention_forward_out(q, q, q, forward, first, n)   # whatever is set up once is set up
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        bm = build_mask(mp, 1, 2, n, n, device=cuda_device)
        torch.cuda._sleep(400_000_000)   # about 0.2 s
        late = side.record_event()
    out = torch.empty_like(q)
    omni_attention_forward_out(q, q, q, out, bm, n)
    same = omni_attention(q, q, q, bm)
    got = bm.partial_block_masks
    torch.cuda.current_stream().synchronize()
    assert not late.query()
    assert torch.equal(out, want) and torch.equal(same, want) and torch.equal(got, pool)
    torch.cuda.synchronize()


def test_every_refusal_is_an_omni_attn_error(cuda_device):
    """Unaligned tensors of whole blocks, forward and backward, and lists whose shapes do not fit each other or q."""
    n, numel = 256, 2 * 256 * 64
    flat = torch.randn(numel + 8, device=cuda_device).half()
    unaligned, q = flat[1:1 + numel].view(1, 2, n, 64), flat[:numel].view(1, 2, n, 64)
    mask = lambda: block_mask_from_row_limits(torch.arange(n).view(1, n), 2)
    bm = mask()
    for call in (omni_attention, omni_attention_autograd):
        with pytest.raises(OmniAttnError, match="aligned"):
            call(unaligned, unaligned, unaligned, bm)
    leaf = q.clone().requires_grad_(True)
    out = omni_attention_autograd(leaf, leaf, leaf, bm)
    with pytest.raises(OmniAttnError, match="aligned"):
        out.backward(unaligned)
    for name, cut in (("block_mask_types", lambda t: t[..., :1]), ("kv_num_blocks", lambda t: t[:, :1]),
                      ("kv_indices", lambda t: t[:, :1])):
        for call in (omni_attention, omni_attention_autograd):
            bad = mask()
            setattr(bad, name, cut(getattr(bad, name)))
            with pytest.raises(OmniAttnError):
                call(q, q, q, bad)


@pytest.mark.parametrize("softcap", [0.0, -1.0, float("nan")])
def test_a_cap_that_is_not_positive_is_none(cuda_device, softcap):
    g = torch.Generator().manual_seed(5)
    bm = block_mask_from_row_limits(_limits(256, 256, g), 1)
    q, k, v = (torch.randn(1, 1, 256, 64, generator=g).half().to(cuda_device) for _ in range(3))
    want = omni_attention(q, k, v, bm)
    assert torch.equal(omni_attention(q, k, v, bm, softcap=softcap), want)
    assert torch.equal(omni_attention_autograd(q, k, v, bm, softcap=softcap), want)
