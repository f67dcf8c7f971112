"""ctypes binding to the in-tree sm_100a kernel library.

The library is `gllm_b200/_C/libgllm_b200.so`, built by `gllm_b200.build` with plain
nvcc (`-gencode arch=compute_100a,code=sm_100a`). It exposes a flat C ABI; every entry
point takes raw device pointers plus the CUDA stream handle and returns 0 on success.

On a GPU box a missing library is a hard error (we never silently fall back to PyTorch
on the product path); on a CPU box `available()` is False and callers use the torch
reference ops in `gllm_b200.ops.ref`.
"""
from __future__ import annotations

import ctypes
import os
from ctypes import POINTER, c_float, c_int, c_int64, c_uint32, c_uint64, c_void_p

import torch

_LIB = None
_LIB_ERR = None

LIB_PATH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "_C",
                        "libgllm_b200.so")

MAX_PEERS = 8


class GemmComm(ctypes.Structure):
    """Mirror of `GemmComm` in csrc/gemm/gemm_bf16.cu."""

    _fields_ = [
        ("a_ready", c_void_p),
        ("a_expected", c_void_p),
        ("m_rot", c_int),
        ("rs_world", c_int),
        ("rs_rank", c_int),
        ("rows_per_rank", c_int),
        ("rs_inc", c_uint32),
        ("peer_out", c_void_p * MAX_PEERS),
        ("peer_cnt", c_void_p * MAX_PEERS),
        ("rs_bcast", c_int),
    ]


def _declare(lib):
    def sig(name, argtypes, restype=c_int):
        fn = getattr(lib, name, None)
        if fn is None:
            return
        fn.argtypes = argtypes
        fn.restype = restype

    P, I, L, F, U = c_void_p, c_int, c_int64, c_float, c_uint32
    sig("gllm_gemm_bf16", [P, L, P, L, P, L, I, I, I, P, I, I, POINTER(GemmComm), P, L, P, I, P])
    sig("gllm_batch_load", [P, P, I, L, P])
    sig("gllm_gemm_bf16_tiles_covering", [I, I, I, I, I, I, I, L, I])
    sig("gllm_gemm_bf16_batched", [P, L, L, P, P, L, L, I, I, I, I, P])
    sig("gllm_gemm_smallm", [P, L, P, L, P, L, I, I, I, P, I, I, P, L, P, P])
    sig("gllm_gemm_bf16_cluster", [P, L, P, L, P, L, I, I, I, P, I, I, I, I, I, P])
    sig("gllm_norm_gemv", [P, L, P, P, P, F, P, L, P, L, I, I, I, P, I, P])
    sig("gllm_rmsnorm", [P, P, P, P, P, I, I, L, F, P])
    sig("gllm_rmsnorm_two", [P, L, P, P, I, P, L, P, P, I, I, F, P])
    sig("gllm_silu_and_mul", [P, P, I, I, L, P])
    sig("gllm_embedding", [P, P, P, I, I, I, I, P])
    sig("gllm_gather_rows", [P, P, P, I, I, P])
    sig("gllm_rope_kv_write",
        [P, L, L, I, P, L, L, I, P, L, L, P, P, P, I, I, I, I, P, P, F, P, P, I, I, I, L, P])
    sig("gllm_attn_decode", [P, L, P, P, P, L, P, P, P, P, I, I, I, I, I, I, I, I, F, P, P])
    sig("gllm_attn_prefill", [P, L, P, P, P, L, P, P, P, I, I, I, I, I, I, I, I, F, P])
    sig("gllm_attn_prefill_tc", [P, L, P, P, P, L, P, P, P, I, I, I, I, I, I, I, I, I, F, I, P])
    sig("gllm_mla_attention", [P, P, P, L, P, P, P, P, P, P, I, I, I, I, I, F, I, P, P])
    sig("gllm_mla_rope_cache", [P, L, L, I, P, L, L, P, L, P, L, P, P, P, P, I, I, P])
    sig("gllm_mla_block_scratch", [I, I, I, I], L)
    sig("gllm_mla_block", [P, L, I, I, I, I, P, P, P, F, P, P, P, P, P, P, P, L, I, P, I, P, F, I, P, P, L, P, L, P, P, I, I, P])
    sig("gllm_mla_gather", [P, P, I, P, P, I, I, I, I, I, P, P, P, P])
    sig("gllm_attn_prefill_expanded", [P, L, P, L, P, P, L, P, P, P, I, I, I, I, I, F, P])
    sig("gllm_sample", [P, I, L, P, I, I, P, P, P, P, P, I, P, c_uint64, P, P, I, P])
    sig("gllm_mark_seen", [P, I, P, P, I, P])
    sig("gllm_vp_candidates", [P, I, L, P, I, I, I, I, P, P, P, P, P, I, P, c_uint64, P, I, P])
    sig("gllm_vp_final", [P, I, I, I, I, P, P, c_uint64, P, P, P])
    sig("gllm_moe_topk_softmax", [P, L, P, P, I, I, I, I, P])
    sig("gllm_moe_grouped_topk", [P, L, P, P, P, I, I, I, I, I, I, I, F, P])
    sig("gllm_moe_align_gather", [P, P, I, I, I, P, P, I, P, P, L, P, I, P, P])
    sig("gllm_moe_grouped_gemm", [P, L, P, P, L, I, I, I, I, P, P, I, P, P])
    sig("gllm_moe_grouped_gemm_glu", [P, L, P, P, L, I, I, I, I, P, P, F, F, P])
    sig("gllm_gemm_bf16_glu", [P, L, P, L, P, L, I, I, I, F, F, P, L, P, I, P])
    sig("gllm_gemm_bf16_gelu", [P, L, P, L, P, L, I, I, I, P, L, P, I, P])
    sig("gllm_moe_align_gather_fp8", [P, P, I, I, I, P, P, I, P, P, L, P, P, I, P])
    sig("gllm_moe_combine", [P, P, P, P, I, I, I, P])
    sig("gllm_fp8_quant_group", [P, L, P, P, I, I, P, P])
    sig("gllm_moe_grouped_gemm_fp8", [P, P, P, P, P, L, I, I, I, I, I, P, P, I, P])
    sig("gllm_set_waits", [P, c_uint32])
    sig("gllm_gemm_fp8_block", [P, P, P, P, P, L, I, I, I, P, I, P])


_NEEDED = None     # csrc groups this process needs (None: all of them)


def require(groups):
    """Called before the first `load()` by an entry point that knows its model: a missing library is then built with
    these kernel families only (csrc sub-directories). A library that holds fewer than needed is completed."""
    global _NEEDED
    _NEEDED = set(groups) if groups is not None else None


def _lacking() -> bool:
    from gllm_b200 import build as _build
    held = _build.built_groups()
    if held is None:
        return False
    need = _build.all_groups() if _NEEDED is None else (_NEEDED & _build.all_groups())
    return not need <= held


def load():
    global _LIB, _LIB_ERR
    if _LIB is not None:
        return _LIB
    if _LIB_ERR is not None:
        raise _LIB_ERR
    try:
        if not os.path.exists(LIB_PATH) or _lacking():
            # safety net: build in-tree on first use when a toolchain is present (takes about a minute); a box
            # without nvcc gets the loud error — there is no PyTorch fallback on the GPU path
            try:
                from gllm_b200 import build as _build
                held = _build.built_groups() if os.path.exists(LIB_PATH) else None
                _build.build(groups=None if _NEEDED is None else (_NEEDED | (held or set())))
            except Exception as be:  # noqa: BLE001
                raise FileNotFoundError(
                    f"{LIB_PATH} not found and the in-tree build failed ({be}) — run `python -m gllm_b200.build` "
                    f"(or __graft_entry__.build())") from be
        lib = ctypes.CDLL(LIB_PATH)
        _declare(lib)
        _LIB = lib
        if torch.cuda.is_initialized():
            watch_waits()
        return lib
    except Exception as e:  # noqa: BLE001
        _LIB_ERR = e
        raise


_WAIT_WORD = None     # (pinned tensor that lives as long as the process, the same word as a numpy array)
WAIT_LIMIT_NS = 2_000_000_000     # below 2^32


def watch_waits(limit_ns: int = WAIT_LIMIT_NS):
    """Gives the kernels with bounded waits (csrc/common/bounded.cuh) the word that they set when a wait ran out, and the
    limit. The word is pinned host memory: reading it needs no copy and no synchronisation beyond that of the step."""
    global _WAIT_WORD
    lib = load()
    if not hasattr(lib, "gllm_set_waits"):
        return                       # a library of other kernel families
    if _WAIT_WORD is None:
        word = torch.zeros(1, dtype=torch.int32, pin_memory=True)
        _WAIT_WORD = (word, word.numpy())
    check(lib.gllm_set_waits(_WAIT_WORD[0].data_ptr(), limit_ns), "set_waits")


def waits_gave_up(clear: bool = False) -> bool:
    """Whether a wait of a kernel that has finished ran out since the last clear."""
    if _WAIT_WORD is None:
        return False
    seen = bool(_WAIT_WORD[1][0])
    if clear:
        _WAIT_WORD[1][0] = 0
    return seen


def raise_if_waits_gave_up():
    if waits_gave_up(clear=True):
        raise RuntimeError("a kernel's bounded wait ran out: the results since the last check are invalid")


def available() -> bool:
    """True iff a CUDA device is present (then the library MUST load)."""
    if not torch.cuda.is_available():
        return False
    load()
    return True


def stream_ptr() -> int:
    """The current stream of the current device. Asked for at every launch: `torch.cuda.current_stream()` builds a stream object
    and looks the device up again, some 5 us of the 10 that an eager launch took."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def check(rc: int, what: str):
    if rc != 0:
        raise RuntimeError(f"gllm_b200 kernel launch failed: {what} (rc={rc})")
