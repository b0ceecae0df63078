"""Host-side operator: ``omni_attention(q, k, v, block_mask)``.

Same contract as the reference's wrappers ``omni_attention_shared_kv`` and siblings
(omni-attn-mma/omni_attn_torch.py:517-671): ``[B, H, N, D]`` inputs, an ``OmniBlockMask``, output
``[B, H, N, D]`` sliced back to the unpadded length. Differences, all deliberate:
  * the input dtype is kept (fp16 or bf16); the reference forces ``.half()`` (:609-611);
  * ``scale`` is honoured; the reference accepts and drops it (:517-523 vs :652-663);
  * the launch goes to torch's current stream and nothing synchronises the device (the reference
    calls ``torch.cuda.synchronize()`` after every launch, :666);
  * ``return_lse=True`` also returns the log-sum-exp rows;
  * mask tensors are converted / bit-packed once per mask object and cached on it;
  * tensors are not padded: the kernels take [B, H, N, D] of any N as it lies in memory.
``omni_attention`` and ``omni_attention_autograd`` go through the in-tree ``omni_attn`` extension module (one
native call per operator call), everything else through the C ABI of ``libomni_attn_sm100.so`` with raw
device pointers. There is no CPU or PyTorch fallback: a missing library or a non-CUDA tensor raises.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import os
import sysconfig
from typing import Optional, Tuple, Union

import torch
from torch import Tensor

from .block_mask import OmniBlockMask, retile_block_mask

_LIB_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "libomni_attn_sm100.so")
_lib = None

# symbols include/omni_attn_sm100.h declares
ABI_SYMBOLS = (
    "omni_attn_fwd_sm100",
    "omni_attn_fwd_scratch_sm100",
    "omni_attn_fwd_ex_sm100",
    "omni_attn_fwd_rows_sm100",
    "omni_attn_fwd_noalloc_sm100",
    "omni_attn_fwd_simple_sm100",
    "omni_attn_pack_partial_masks_sm100",
    "omni_attn_pack_partial_masks_blk_sm100",
    "omni_attn_max_seqlen",
    "omni_attn_set_wait_cycles",
    "omni_attn_build_mask_sm100",
    "omni_attn_bwd_workspace_bytes",
    "omni_attn_bwd_sm100",
    "omni_attn_bwd_ex_sm100",
    "omni_attn_bwd_rows_sm100",
    "omni_attn_error_string",
    "omni_attn_last_cuda_error",
    "omni_attn_abi_version",
)

SCRATCH_BYTES = 256  # OMNI_ATTN_SCRATCH_BYTES
STATUS_WAIT_TIMEOUT = 1
STATUS_BAD_INDEX = 2


class OmniAttnError(RuntimeError):
    """A C-ABI call returned an error code, or a kernel reported a bad status."""


def load_library() -> ctypes.CDLL:
    """Load libomni_attn_sm100.so from the package directory (built by ``omni_attention_b200.build``);
    the environment variable OMNI_ATTN_LIBRARY names another build of the same library, which the extension module
    then calls too."""
    global _lib
    if _lib is not None:
        return _lib
    path = os.environ.get("OMNI_ATTN_LIBRARY", _LIB_PATH)
    if not os.path.exists(path):
        raise ImportError(
            f"{path} not found: build it with `python -m omni_attention_b200.build` "
            "(there is no fallback implementation)")
    lib = ctypes.CDLL(path)
    vp, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    fwd_args = [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp] + [i32] * 10 + [f32, vp, vp]
    for name in ("omni_attn_fwd_sm100", "omni_attn_fwd_simple_sm100", "omni_attn_fwd_noalloc_sm100"):
        fn = getattr(lib, name)
        fn.argtypes = fwd_args
        fn.restype = i32
    lib.omni_attn_fwd_scratch_sm100.argtypes = fwd_args + [vp, ctypes.c_longlong]
    lib.omni_attn_fwd_scratch_sm100.restype = i32
    lib.omni_attn_fwd_ex_sm100.argtypes = fwd_args + [f32, vp, ctypes.c_longlong]
    lib.omni_attn_fwd_ex_sm100.restype = i32
    lib.omni_attn_pack_partial_masks_sm100.argtypes = [vp, vp, i32, vp]
    lib.omni_attn_pack_partial_masks_sm100.restype = i32
    lib.omni_attn_pack_partial_masks_blk_sm100.argtypes = [vp, vp, i32, i32, vp]
    lib.omni_attn_pack_partial_masks_blk_sm100.restype = i32
    lib.omni_attn_max_seqlen.argtypes = [i32, i32, i32]
    lib.omni_attn_max_seqlen.restype = i32
    lib.omni_attn_set_wait_cycles.argtypes = [ctypes.c_longlong]
    lib.omni_attn_set_wait_cycles.restype = None
    lib.omni_attn_build_mask_sm100.argtypes = [vp, i32, i32, i32, i32, i32, vp, vp, vp, vp, vp, vp, i32, vp, vp,
                                               ctypes.c_longlong, vp]
    lib.omni_attn_build_mask_sm100.restype = i32
    lib.omni_attn_bwd_workspace_bytes.argtypes = [i32, i32, i32]
    lib.omni_attn_bwd_workspace_bytes.restype = ctypes.c_longlong
    lib.omni_attn_bwd_sm100.argtypes = [vp] * 15 + [i32] * 10 + [f32, vp, vp, vp, ctypes.c_longlong]
    lib.omni_attn_bwd_sm100.restype = i32
    lib.omni_attn_bwd_ex_sm100.argtypes = lib.omni_attn_bwd_sm100.argtypes + [f32]
    lib.omni_attn_bwd_ex_sm100.restype = i32
    lib.omni_attn_error_string.argtypes = [i32]
    lib.omni_attn_error_string.restype = ctypes.c_char_p
    lib.omni_attn_last_cuda_error.argtypes = []
    lib.omni_attn_last_cuda_error.restype = i32
    lib.omni_attn_abi_version.argtypes = []
    lib.omni_attn_abi_version.restype = i32
    _lib = lib
    return lib


def _check(rc: int) -> None:
    if rc != 0:
        lib = load_library()
        msg = lib.omni_attn_error_string(rc).decode()
        extra = f", CUDA error {lib.omni_attn_last_cuda_error()}" if rc == -10 else ""
        raise OmniAttnError(f"omni_attn: {msg} (code {rc}{extra})")


def _ptr(t: Optional[Tensor]) -> Optional[int]:
    return None if t is None or t.numel() == 0 else t.data_ptr()


def pack_partial_masks(partial_block_masks: Tensor) -> Tensor:
    """[P, blk, blk] bool (CUDA; blk = 128 or 64) -> [P, blk, blk / 32] int32 bit masks, on the current stream."""
    assert partial_block_masks.is_cuda and partial_block_masks.dtype == torch.bool
    P, blk = partial_block_masks.shape[0], int(partial_block_masks.shape[1])
    if blk not in (64, 128) or partial_block_masks.shape[2] != blk:
        raise OmniAttnError(f"partial_block_masks must be [P, 64, 64] or [P, 128, 128], got {tuple(partial_block_masks.shape)}")
    src = partial_block_masks.contiguous()
    bits = torch.empty(P, blk, blk // 32, dtype=torch.int32, device=src.device)
    if P > 0:
        with torch.cuda.device(src.device):
            stream = torch.cuda.current_stream().cuda_stream
            _check(load_library().omni_attn_pack_partial_masks_blk_sm100(src.data_ptr(), bits.data_ptr(), P, blk, stream))
    return bits


def build_block_mask_cuda(modality_positions: Tensor, batch: int, nheads: int, seq_len: int, padded: int,
                          device: torch.device) -> OmniBlockMask:
    """Runs omni_attn_build_mask_sm100 on ``device`` and wraps its outputs in an OmniBlockMask whose
    tensors stay on the device. Nothing here waits for the GPU: the pool of PARTIAL tiles is sized by what a
    sequence of that many blocks can need at most. The kernel writes the pool bit-packed, which is what the
    attention kernels read; the container's byte-per-element ``partial_block_masks`` is expanded from it
    only if somebody reads that field."""
    res = load_extension().build_mask(modality_positions, batch, nheads, int(seq_len), int(padded),
                               device.index if device.index is not None else torch.cuda.current_device())
    if isinstance(res, int):
        _check(res)
    mask, nb, idx, typ, pidx, bits, count = res
    device = nb.device
    bm = OmniBlockMask(nb, idx, typ, padded, padded, 128, 128, pidx, None)

    def expand_pool() -> Tensor:
        # first read of the reference-shaped pool: waits for the GPU to learn how many tiles there are
        mask.order_after_build()
        need = int(count.item())
        if need > bits.shape[0]:
            raise OmniAttnError(f"mask builder: {need} PARTIAL tiles in a pool of {bits.shape[0]}")
        shifts = torch.arange(32, dtype=torch.int32, device=device)
        return ((bits[:need].unsqueeze(-1) >> shifts) & 1).bool().view(need, 128, 128)

    bm.set_lazy_partial_pool(expand_pool)
    bm._cache[device.index] = mask
    # what omni_attention_forward_out uses; a caller that asks for the byte-per-element pool
    # (pack_bits=False) gets it through the container's field, expanded then
    bm._cache[(str(device), True)] = {"nb": nb, "idx": idx, "typ": typ, "pidx": pidx, "pbool": None, "pbits": bits,
                                      "num_partial": int(bits.shape[0]), "order_after_build": mask.order_after_build}
    return bm


def _device_mask(bm: OmniBlockMask, device: torch.device, pack_bits: bool) -> dict:
    """int32 contiguous copies of the mask tensors on ``device`` (+ bit-packed pool), cached on the mask."""
    key = (str(device), pack_bits)
    hit = bm._cache.get(key)
    if hit is not None:
        # The copies and the pack kernel were enqueued on the stream that was current when the entry
        # was built; a call on another stream must not run ahead of them.
        hit["order_after_build"]()
        return hit
    cv = lambda t: t.to(device=device, dtype=torch.int32).contiguous()
    d = {"nb": cv(bm.kv_num_blocks), "idx": cv(bm.kv_indices), "typ": cv(bm.block_mask_types),
         "pidx": None, "pbool": None, "pbits": None, "num_partial": 0}
    if bm.partial_block_mask_indices is not None and bm.partial_block_masks is not None:
        d["pidx"] = cv(bm.partial_block_mask_indices)
        pool = bm.partial_block_masks.to(device=device, dtype=torch.bool).contiguous()
        d["num_partial"] = int(pool.shape[0])
        if pool.shape[0] > 0:
            if pack_bits:
                d["pbits"] = pack_partial_masks(pool)
            else:
                d["pbool"] = pool
    with torch.cuda.device(device):
        built_on, ready = torch.cuda.current_stream(device), torch.cuda.Event()
        ready.record(built_on)

    def order_after_build():
        cur = torch.cuda.current_stream(device)
        if cur != built_on:
            cur.wait_event(ready)

    d["order_after_build"] = order_after_build
    bm._cache[key] = d
    return d


_ext = None


def load_extension():
    """The in-tree extension module (built by ``omni_attention_b200.build``). It is loaded by its path and kept here:
    the operator neither reads nor sets ``sys.modules["omni_attn"]``, where a program may have the reference's own
    extension (``install_reference_module`` registers this one there for those who ask)."""
    global _ext
    if _ext is None:
        path = os.path.join(os.path.dirname(_LIB_PATH), "omni_attn" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
        if not os.path.exists(path):
            raise ImportError(f"{path} not found: build it with `python -m omni_attention_b200.build`")
        spec = importlib.util.spec_from_file_location("omni_attn", path)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        lib = load_library()._name
        if os.path.realpath(lib) != os.path.realpath(_LIB_PATH):   # OMNI_ATTN_LIBRARY
            mod.use_library(os.path.abspath(lib))
        mod.set_error_type(OmniAttnError)
        _ext = mod
    return _ext


def _native_mask(bm: OmniBlockMask, device: torch.device):
    """The mask in the extension module's form, made once per mask object and device; None for a mask or a
    device it does not take, which the caller's own checks then name."""
    if device.type != "cuda" or bm.Q_BLOCK_SIZE not in (64, 128) or bm.KV_BLOCK_SIZE != bm.Q_BLOCK_SIZE or bm.kv_len != bm.q_len:
        return None
    d = _device_mask(bm, device, True)
    mask = load_extension().DeviceMask(d["nb"], d["idx"], d["typ"], d["pidx"], d["pbool"], d["pbits"], d["num_partial"],
                                bm.Q_BLOCK_SIZE, bm.q_len)
    bm._cache[device.index] = mask
    return mask


def omni_attention_forward_out(q: Tensor, k: Tensor, v: Tensor, out: Tensor, block_mask: OmniBlockMask,
                               seqlen_orig: int, scale: Optional[float] = None, lse: Optional[Tensor] = None,
                               status: Optional[Tensor] = None, kernel: str = "ws", pack_bits: bool = True,
                               softcap: Optional[float] = None) -> None:
    """Launch the forward on padded, contiguous CUDA tensors; writes ``out`` (and ``lse``) in place."""
    _check_tensors(q, k, v, out)
    B, H, N, D = q.shape
    m = _device_mask(block_mask, q.device, pack_bits)
    nq = N // block_mask.Q_BLOCK_SIZE if block_mask.Q_BLOCK_SIZE else 0
    if tuple(m["nb"].shape) != (B, H, nq):
        raise OmniAttnError(f"kv_num_blocks shape {tuple(m['nb'].shape)} != {(B, H, nq)}")
    if tuple(m["idx"].shape[:3]) != (B, H, nq) or m["typ"].shape != m["idx"].shape:
        raise OmniAttnError("kv_indices / block_mask_types shape mismatch")
    if m["pidx"] is not None and m["pidx"].shape != m["idx"].shape:
        raise OmniAttnError("partial_block_mask_indices shape mismatch")
    if lse is not None and (lse.dtype != torch.float32 or lse.numel() != B * H * N or not lse.is_contiguous()):
        raise OmniAttnError("lse must be contiguous float32 [B, H, N]")
    lib = load_library()
    if kernel not in ("ws", "ws_static", "simple"):
        raise OmniAttnError(f"unknown kernel {kernel!r}")
    with torch.cuda.device(q.device):
        stream = torch.cuda.current_stream().cuda_stream
        args = (q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), _ptr(lse), m["nb"].data_ptr(),
                m["idx"].data_ptr(), m["typ"].data_ptr(), _ptr(m["pidx"]), _ptr(m["pbool"]), _ptr(m["pbits"]),
                B, H, N, int(seqlen_orig), D, block_mask.Q_BLOCK_SIZE, block_mask.KV_BLOCK_SIZE,
                int(m["idx"].shape[3]), m["num_partial"], 1 if q.dtype == torch.bfloat16 else 0,
                float(scale) if scale is not None else 0.0, stream, _ptr(status))
        if softcap is not None and softcap > 0:
            if kernel == "simple":
                raise OmniAttnError("the plain kernel has no soft-cap")
            sc = _scratch_for(q.device, stream) if kernel == "ws" else None
            rc = lib.omni_attn_fwd_ex_sm100(*args, float(softcap), _ptr(sc), SCRATCH_BYTES if sc is not None else 0)
        elif kernel == "ws":
            # dynamic unit hand-out: one small scratch buffer per (device, stream), reused by every
            # call on that stream (calls on one stream never overlap)
            rc = lib.omni_attn_fwd_scratch_sm100(*args, _scratch_for(q.device, stream).data_ptr(), SCRATCH_BYTES)
        elif kernel == "ws_static":
            rc = lib.omni_attn_fwd_sm100(*args)
        else:
            rc = lib.omni_attn_fwd_simple_sm100(*args)
    _check(rc)


_scratch = {}


def _scratch_for(device: torch.device, stream: int) -> Tensor:
    key = (str(device), int(stream))
    t = _scratch.get(key)
    if t is None:
        t = torch.zeros(SCRATCH_BYTES // 4, dtype=torch.int32, device=device)
        _scratch[key] = t
    return t


def _pad_to_block(x: Tensor, block: int) -> Tensor:
    rem = (-x.shape[2]) % block
    return (x if rem == 0 else torch.nn.functional.pad(x, (0, 0, 0, rem))).contiguous()


def _check_shapes(query: Tensor, key: Tensor, value: Tensor, block_mask: OmniBlockMask) -> None:
    """What the operator asks of its arguments, as errors (the reference launchers' checks,
    omni-attn-mma/mma/omni_attn_shared_kv.cu:725-741: head_dim 32/64/128, blocks 64 or 128)."""
    B, H, Q, D = query.shape
    if key.shape != (B, H, Q, D) or value.shape != (B, H, Q, D):
        raise OmniAttnError(f"key/value shape must equal query shape {(B, H, Q, D)} (Q_len == KV_len)")
    if D not in (32, 64, 128):
        raise ValueError(f"Unsupported head_dim={D}. Supported: 32, 64, 128.")
    if (block_mask.Q_BLOCK_SIZE, block_mask.KV_BLOCK_SIZE) not in ((64, 64), (128, 128)):
        raise ValueError("Unsupported block size: Q_BLOCK_SIZE and KV_BLOCK_SIZE must both be 64 or both be 128.")
    padded = -(-Q // block_mask.Q_BLOCK_SIZE) * block_mask.Q_BLOCK_SIZE
    if padded != block_mask.q_len or padded != block_mask.kv_len:
        raise OmniAttnError(
            f"padded length {padded} does not match the mask's q_len/kv_len ({block_mask.q_len}/{block_mask.kv_len})")


def _check_tensors(q: Tensor, k: Tensor, v: Tensor, out: Tensor, need_contiguous: bool = True) -> None:
    if not (q.is_cuda and k.is_cuda and v.is_cuda and out.is_cuda):
        raise OmniAttnError("omni_attention needs CUDA tensors (there is no CPU path)")
    if q.dtype not in (torch.float16, torch.bfloat16):
        raise OmniAttnError(f"unsupported dtype {q.dtype}: fp16 or bf16")
    for t in (k, v, out):
        if t.dtype != q.dtype or t.shape != q.shape or t.device != q.device:
            raise OmniAttnError("q, k, v, out must share dtype, shape and device (Q_len == KV_len)")
    for t in (q, k, v, out):
        if need_contiguous and not t.is_contiguous():
            raise OmniAttnError("q, k, v, out must be contiguous")


def _cap(softcap: Optional[float]) -> float:
    """The native calls' form of ``softcap``: 0 = none, which is also what a value that is not positive means."""
    return float(softcap) if softcap is not None and softcap > 0 else 0.0


def _refuse(query: Tensor, key: Tensor, value: Tensor, block_mask: OmniBlockMask) -> None:
    """Names what is wrong with a call the extension module did not take."""
    _check_shapes(query, key, value, block_mask)
    _check_tensors(query, key, value, query, need_contiguous=False)
    raise OmniAttnError(f"kv_num_blocks shape {tuple(block_mask.kv_num_blocks.shape)} does not fit q {tuple(query.shape)}")


def omni_attention(query: Tensor, key: Tensor, value: Tensor, block_mask: OmniBlockMask,
                   scale: Optional[float] = None, return_lse: bool = False, kernel: str = "ws",
                   check_status: bool = False, softcap: Optional[float] = None) -> Union[Tensor, Tuple[Tensor, Tensor]]:
    """Block-mask attention forward on a B200.

    query/key/value: [B, H, N, D] fp16 or bf16 CUDA tensors with Q_len == KV_len, D in {32, 64, 128};
    ``block_mask`` with 128x128 or 64x64 blocks, built for the length padded to its block size. Returns ``out[:, :, :N]`` (and
    ``lse[:, :, :N]``, natural log, when ``return_lse``). ``softcap`` > 0 applies the Transfusion attention's
    tanh soft-cap to the scaled scores before masking (transfusion_pytorch/transfusion.py:358-364). ``check_status=True`` synchronises and
    raises if the kernel reported a bounded-wait timeout or an out-of-range block index.
    """
    if kernel == "ws" and not check_status:
        mask = block_mask._cache.get(query.get_device())
        if mask is None:
            mask = _native_mask(block_mask, query.device)
        res = None
        if mask is not None:
            res = load_extension().operator_forward(mask, query, key, value, scale or 0.0, _cap(softcap), return_lse)
        if res is None:
            _refuse(query, key, value, block_mask)
        if isinstance(res, int):
            _check(res)
        return res
    # the plain kernel, the fixed unit assignment, the status word: padded as the C ABI's basic entries want it
    _check_shapes(query, key, value, block_mask)
    B, H, n_orig = query.shape[:3]
    qp, kp, vp = (_pad_to_block(t, block_mask.Q_BLOCK_SIZE) for t in (query, key, value))
    out = torch.empty_like(qp)
    lse = torch.empty(B, H, qp.shape[2], dtype=torch.float32, device=qp.device) if return_lse else None
    status = torch.zeros(1, dtype=torch.int32, device=qp.device) if check_status else None
    omni_attention_forward_out(qp, kp, vp, out, block_mask, n_orig, scale, lse, status, kernel, softcap=softcap)
    if check_status:
        code = int(status.item())
        if code & 0xFF == STATUS_WAIT_TIMEOUT:
            raise OmniAttnError(f"kernel gave up waiting (status {code:#x}); output is not valid")
        if code & 0xFF == STATUS_BAD_INDEX:
            raise OmniAttnError("kv_indices holds a block id outside [0, num_kv_blocks); the entry was skipped")
    out = out[:, :, :n_orig]
    if return_lse:
        return out, lse[:, :, :n_orig]
    return out


def omni_attention_backward_out(q: Tensor, k: Tensor, v: Tensor, out: Tensor, lse: Tensor, d_out: Tensor,
                                dq: Tensor, dk: Tensor, dv: Tensor, block_mask: OmniBlockMask, seqlen_orig: int,
                                scale: Optional[float] = None, status: Optional[Tensor] = None,
                                workspace: Optional[Tensor] = None, softcap: Optional[float] = None) -> None:
    """Launch the backward on padded, contiguous CUDA tensors; writes ``dq``, ``dk``, ``dv`` in place.
    ``out`` and ``lse`` are what the forward returned for the same inputs, mask and scale. The
    reference has no backward; this is the gradient of its forward definition. ``softcap`` must be
    the value the forward was run with."""
    tensors = (q, k, v, out, d_out, dq, dk, dv)
    if not all(t.is_cuda for t in tensors) or not lse.is_cuda:
        raise OmniAttnError("omni_attention backward needs CUDA tensors (there is no CPU path)")
    if q.dtype not in (torch.float16, torch.bfloat16):
        raise OmniAttnError(f"unsupported dtype {q.dtype}: fp16 or bf16")
    for t in tensors:
        if t.dtype != q.dtype or t.shape != q.shape or not t.is_contiguous():
            raise OmniAttnError("q, k, v, out, d_out, dq, dk, dv must be contiguous and share dtype and shape")
    B, H, N, D = q.shape
    if lse.dtype != torch.float32 or lse.numel() != B * H * N or not lse.is_contiguous():
        raise OmniAttnError("lse must be contiguous float32 [B, H, N]")
    m = _device_mask(block_mask, q.device, True)
    lib = load_library()
    need = int(lib.omni_attn_bwd_workspace_bytes(B, H, N))
    if workspace is None:
        workspace = torch.empty(need, dtype=torch.uint8, device=q.device)
    with torch.cuda.device(q.device):
        stream = torch.cuda.current_stream().cuda_stream
        args = (q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), d_out.data_ptr(),
                dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), m["nb"].data_ptr(), m["idx"].data_ptr(),
                m["typ"].data_ptr(), _ptr(m["pidx"]), _ptr(m["pbool"]), _ptr(m["pbits"]), B, H, N, int(seqlen_orig), D,
                block_mask.Q_BLOCK_SIZE, block_mask.KV_BLOCK_SIZE, int(m["idx"].shape[3]), m["num_partial"],
                1 if q.dtype == torch.bfloat16 else 0, float(scale) if scale is not None else 0.0, stream,
                _ptr(status), workspace.data_ptr(), workspace.numel() * workspace.element_size())
        if softcap is not None and softcap > 0:
            rc = lib.omni_attn_bwd_ex_sm100(*args, float(softcap))
        else:
            rc = lib.omni_attn_bwd_sm100(*args)
    _check(rc)


def omni_attention_autograd(query: Tensor, key: Tensor, value: Tensor, block_mask: OmniBlockMask,
                            scale: Optional[float] = None, softcap: Optional[float] = None) -> Tensor:
    """``omni_attention`` for training: same inputs and output, differentiable with respect to
    query, key and value (the gradients come from omni_attn_bwd_sm100 / omni_attn_bwd_ex_sm100)."""
    if block_mask.Q_BLOCK_SIZE == 64 and block_mask.KV_BLOCK_SIZE == 64:
        # the backward kernels take 128-blocks: re-expressed quadrant by quadrant, once per mask object
        hit = block_mask._cache.get("retiled128")
        if hit is None:
            hit = block_mask._cache["retiled128"] = retile_block_mask(block_mask, 128)
        block_mask = hit
    mask = block_mask._cache.get(query.get_device())
    if mask is None:
        mask = _native_mask(block_mask, query.device)
    out = None
    if mask is not None:
        out = load_extension().operator_autograd(mask, query, key, value, scale or 0.0, _cap(softcap))
    if out is None:
        _refuse(query, key, value, block_mask)
    return out


def default_scale(head_dim: int) -> float:
    return 1.0 / math.sqrt(head_dim)
