"""What a user of this package has it do: block-mask attention, forward and training, through the
public entry points, from a 512-token sequence to one GPU's share of a 32K-token batch.

A case is one pass of a user's program:

  op = "fwd"         omni_attention(q, k, v, mask): prefill / scoring with a mask that is kept
       "train"       omni_attention_autograd and the gradients of q, k, v
       "model"       one forward of a Transfusion-style model: the mask built from the spans of the
                     batch, then the attention core of each layer with the tanh soft-cap
       "model_train" the same with the gradients of every layer's q, k, v
       "module"      the reference's 13-argument binding, called as the reference's wrapper calls it:
                     a fresh output, int32 lists, the byte-per-element mask pool

  pattern = "causal"  plain causal text
            "random"  skipped / FULL / PARTIAL (Bernoulli element mask) blocks below a CAUSAL diagonal
            "image256", "image1024", "multi"  causal text with images attended in both directions:
                      256-token images, 4-6 images of 1024, 8-16 images of 256 / 1024 / 4096

N is the length before padding to the block size; the layout of the images, the random blocks, Q, K, V
and the incoming gradient all come from the seed.
"""
import math
import random

import torch

import omni_attention_b200 as omni
from omni_attention_b200.inputs import random_fcp_block_mask
from omni_attention_b200.transfusion import transfusion_attention_core, transfusion_block_mask

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
SOFTCAP = 50.0   # the Transfusion model's default
LARGEST_FLOPS = 2.5e12   # of a drawn case; the largest listed one has about twice that


def _case(name, op, pattern, B, H, N, D, dtype, block=128, lse=False, layers=1):
    c = dict(op=op, pattern=pattern, B=B, H=H, N=N, D=D, dtype=dtype, block=block, lse=lse, layers=layers)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short prompt: the launch and the host path are all there is
        _case("fwd causal 512", "fwd", "causal", 1, 8, 512, 64, "fp16"),
        # every block type in one mask, the log-sum-exp kept (for merging with other attention parts)
        _case("fwd random 2048 lse", "fwd", "random", 1, 8, 2048, 64, "fp16", lse=True),
        # a batch of interleaved text and small images at head_dim 64
        _case("fwd image256 4096", "fwd", "image256", 2, 16, 4096, 64, "bf16"),
        # the headline workload: a vision-language prefill at head_dim 128
        _case("fwd image1024 8192", "fwd", "image1024", 1, 32, 8192, 128, "bf16"),
        # one eighth of a 4 x 32-head batch of 32K tokens: what one of eight GPUs owns
        _case("fwd multi 32768", "fwd", "multi", 1, 16, 32768, 128, "bf16"),
        # 64 x 64 blocks and a length that is no multiple of anything
        _case("fwd blocks64 ragged 1999", "fwd", "image256", 2, 16, 1999, 128, "bf16", block=64),
        # the narrowest head, short
        _case("fwd head_dim 32 448", "fwd", "random", 2, 8, 448, 32, "fp16", block=64),
        # the reference's own binding, fp16 as its wrapper forces
        _case("module image1024 4096", "module", "image1024", 1, 16, 4096, 128, "fp16"),
        # inference through a small Transfusion model: mask and four layers
        _case("model image256 2048", "model", "image256", 2, 8, 2048, 64, "bf16", layers=4),
        # its training step on a ragged batch
        _case("model_train image256 1500", "model_train", "image256", 2, 8, 1500, 64, "bf16", layers=2),
        # training at head_dim 64 and at the headline sizes
        _case("train image256 4096", "train", "image256", 2, 16, 4096, 64, "bf16"),
        _case("train image1024 8192", "train", "image1024", 1, 32, 8192, 128, "bf16"),
    ]


def draw(rng):
    """One more case of the same ranges: 100 to 32768 tokens, 1 to 64 (batch, head) pairs."""
    op = rng.choices(["fwd", "train", "model", "model_train", "module"], [5, 4, 2, 2, 1])[0]
    D = rng.choices([32, 64, 128], [1, 3, 4])[0]
    dtype = "fp16" if op == "module" else rng.choice(["fp16", "bf16", "bf16"])
    block = 64 if op in ("fwd", "module") and rng.random() < 0.25 else 128
    layers = rng.randint(1, 4) if op.startswith("model") else 1
    while True:
        N = int(round(math.exp(rng.uniform(math.log(100), math.log(32768)))))
        if op == "module" or rng.random() < 0.3:
            N = -(-N // block) * block   # its callers pad; others often bring whole blocks too
        B, H = rng.choice([1, 1, 2, 4]), rng.choice([4, 8, 12, 16, 32])
        patterns = ["image256"]
        if N >= 4096:
            patterns += ["image1024"]
        if N >= 12288:
            patterns += ["multi"]
        if not op.startswith("model"):
            patterns += ["causal"] + (["random"] if N <= 4096 else [])
        c = _case(None, op, rng.choice(patterns), B, H, N, D, dtype, block, op == "fwd" and rng.random() < 0.3, layers)
        if B * H <= 64 and work(c)["flops"] <= LARGEST_FLOPS:
            return c


def _spans(pattern, N, rng):
    """(offset, length) of the images of one sequence."""
    text, sizes, count = {"image256": ((64, 512), (256,), 1 << 30),
                          "image1024": ((128, 1024), (1024,), rng.randint(4, 6)),
                          "multi": ((256, 2048), (256, 1024, 4096), rng.randint(8, 16))}[pattern]
    spans, pos = [], 0
    while len(spans) < count:
        pos += rng.randint(*text)
        size = rng.choice(sizes)
        if pos + size > N:
            break
        spans.append((pos, size))
        pos += size
    return spans


def _modalities(case, rng, device):
    """[B, M, 3] (type, offset, length), shorter lists filled up with empty spans."""
    per = [_spans(case["pattern"], case["N"], rng) for _ in range(case["B"])]
    m = max(1, max(len(s) for s in per))
    rows = [[(0, o, n) for o, n in s] + [(0, 0, 0)] * (m - len(s)) for s in per]
    return torch.tensor(rows, dtype=torch.int32, device=device)


def _mask(case, seed, rng, device):
    B, H, N, block = case["B"], case["H"], case["N"], case["block"]
    padded = -(-N // block) * block
    if case["pattern"] == "causal":
        return omni.create_causal_omni_block_mask(B, H, N, N, block, block, device)
    if case["pattern"] == "random":
        return random_fcp_block_mask(B, H, padded, seed, block=block).to(device)
    if block == 128 and case["op"] != "module":
        return omni.create_omni_block_mask_from_modality_positions(_modalities(case, rng, device), B, H, N, N, device=device)
    spans = [_spans(case["pattern"], N, rng) for _ in range(B)]
    limits, causal = omni.row_limits_from_modality_positions(padded, spans, device)
    # the reference's masks carry a copy of every PARTIAL tile for each head
    return omni.block_mask_from_row_limits(limits, H, causal, block, share_partial_across_heads=case["op"] != "module")


def prepare(case, seed):
    dev = torch.device("cuda")
    rng = random.Random(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    shape = (case["B"], case["H"], case["N"], case["D"])
    scale = 0.5 if case["D"] == 128 else 1.0
    dtype = DTYPES[case["dtype"]]
    new = lambda s: (torch.randn(shape, generator=gen, device=dev) * s).to(dtype)
    training = case["op"].endswith("train")
    layers = []
    for _ in range(case["layers"]):
        qkv = [new(scale).requires_grad_(training) for _ in range(3)]
        layers.append((*qkv, new(1.0) if training else None))
    state = {"case": case, "layers": layers}
    if case["op"].startswith("model"):
        state["modalities"] = _modalities(case, rng, dev)
        return state
    mask = state["mask"] = _mask(case, seed, rng, dev)
    if case["op"] == "module":
        state["module"] = omni.install_reference_module()
        has_partial = mask.partial_block_mask_indices is not None and mask.partial_block_masks.numel() > 0
        idx = mask.partial_block_mask_indices if has_partial else torch.empty(0, dtype=torch.int32, device=dev)
        pool = mask.partial_block_masks if has_partial else torch.empty(0, dtype=torch.bool, device=dev)
        state["args"] = (mask.kv_num_blocks, mask.kv_indices, mask.block_mask_types, case["block"], case["block"],
                         case["N"], idx, pool, has_partial)
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "fwd":
        q, k, v, _ = state["layers"][0]
        return omni.omni_attention(q, k, v, state["mask"], return_lse=case["lse"])
    if op == "module":
        q, k, v, _ = state["layers"][0]
        out = torch.empty_like(q)
        state["module"].omni_attn_mma_stages_split_q_shared_kv(q, k, v, out, *state["args"])
        return out
    if op == "train":
        q, k, v, d_out = state["layers"][0]
        out = omni.omni_attention_autograd(q, k, v, state["mask"])
        return [out, *torch.autograd.grad(out, (q, k, v), d_out)]
    mask = transfusion_block_mask(state["modalities"], case["H"], case["N"])
    outs = [transfusion_attention_core(q, k, v, mask, SOFTCAP) for q, k, v, _ in state["layers"]]
    if op == "model":
        return outs
    leaves = [t for q, k, v, _ in state["layers"] for t in (q, k, v)]
    return [*outs, *torch.autograd.grad(outs, leaves, [d for *_, d in state["layers"]])]


def _pairs(case):
    """(query, key) pairs of one (batch, head) that attend, of the layout of seed 0 (another seed's layout
    has a few per cent more or fewer). The element masks of random blocks have no structure that could
    be skipped: such a block counts whole."""
    N, block = case["N"], case["block"]
    causal = N * (N + 1) / 2
    if case["pattern"] == "causal":
        return causal
    if case["pattern"] == "random":
        nq = -(-N // block)
        return nq * block * (block + 1) / 2 + 0.8 * nq * (nq - 1) / 2 * block * block
    rng = random.Random(0)
    per = [_spans(case["pattern"], N, rng) for _ in range(case["B"])]
    return causal + sum(n * (n - 1) / 2 for spans in per for _, n in spans) / len(per)


def work(case):
    """Q, K, V (and dO) read once, the output (and dQ, dK, dV) written once; two contractions over the
    attending pairs forward and five backward, whatever is recomputed on the way."""
    training = case["op"].endswith("train")
    bh = case["B"] * case["H"]
    tensors = 8 if training else 4
    flops = (14 if training else 4) * case["D"] * _pairs(case) * bh
    data = tensors * bh * case["N"] * case["D"] * 2 + (4 * bh * case["N"] if case["lse"] else 0)
    return {"bytes": case["layers"] * data, "flops": case["layers"] * flops}


def tolerance(case):
    """The probabilities, dS and the results are rounded to the 16-bit type: 2^-9 (bf16) or 2^-12 (fp16)
    of the value each, a few of them along the way."""
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
