"""ctypes binding of the in-tree sm_100a library (``_lib/libpithb200.so``).

The library has a plain C ABI (raw device pointers + a CUDA stream handle), so it is loaded with
ctypes rather than through torch's extension machinery: builds take seconds and the shared object
travels with the source tree. :func:`lib` raises if the library is missing, so a GPU run can never
silently fall back to eager PyTorch.
"""

from __future__ import annotations

import ctypes
import importlib.util
import sys
import types
from ctypes import c_int, c_longlong, c_void_p, c_float
from functools import lru_cache
from pathlib import Path

import torch

# PITHTRAIN_CHECKED_LIB=1 loads the bounds-checking build (python -m pithtrain_b200.build --bounds-check): a
# diagnostic like a sanitizer run, slower, same entry points.
_LIB_PATH = Path(__file__).resolve().parent / "_lib" / (
    "libpithb200_checked.so" if __import__("os").environ.get("PITHTRAIN_CHECKED_LIB") == "1" else "libpithb200.so")


class NativeLibraryMissing(RuntimeError):
    pass


class KernelStatusError(RuntimeError):
    """A kernel reported a bounded-wait timeout or a capacity overflow through the status word."""


STATUS_NAMES = {
    1: "timeout in TMA producer",
    2: "timeout in MMA issuer",
    3: "timeout in epilogue",
    4: "timeout waiting for a peer",
    5: "receive-buffer capacity exceeded",
    6: "timeout draining in-flight copies",
    7: "dynamic shared memory not 1024-byte aligned",
    8: "index out of bounds (bounds-checking build)",
}


def available() -> bool:
    return _LIB_PATH.exists()


@lru_cache(maxsize=1)
def lib() -> ctypes.CDLL:
    if not _LIB_PATH.exists():
        raise NativeLibraryMissing(
            f"{_LIB_PATH} not found: run `python -m pithtrain_b200.build` (or __graft_entry__.build())"
        )
    L = ctypes.CDLL(str(_LIB_PATH))
    _declare(L)
    return L


_HOST_PATH = _LIB_PATH.with_name("pith_host_ops.so")


@lru_cache(maxsize=1)
def host():
    """The operators whose host side is C++ (``csrc/host_ops.cpp``), bound to the kernels of :func:`lib`."""
    lib()
    if not _HOST_PATH.exists():
        raise NativeLibraryMissing(f"{_HOST_PATH} not found: run `python -m pithtrain_b200.build` (or __graft_entry__.build())")
    spec = importlib.util.spec_from_file_location("pith_host_ops", _HOST_PATH)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    module.bind(str(_LIB_PATH))
    return module


class _TracedStep(torch.autograd.Function):
    """A host operator as one step of a ``torch.jit.trace``. The tracer sees the allocations of a C++ operator, but not its kernels: a
    trace of them alone would replay as unwritten memory. A Python function it records as a call."""

    @staticmethod
    def forward(ctx, op, *args):
        needed = ctx.needs_input_grad[1:]
        ctx.inputs = [a if a.is_leaf else a.detach().requires_grad_() for a, grad in zip(args, needed) if grad]
        leaves = iter(ctx.inputs)
        with torch.set_grad_enabled(bool(ctx.inputs)):
            outs = op(*(next(leaves) if grad else a for a, grad in zip(args, needed)))
        ctx.outs = outs if isinstance(outs, tuple) else (outs,)
        ctx.set_materialize_grads(False)
        given = tuple(None if o is None else o.detach() for o in ctx.outs)
        ctx.mark_non_differentiable(*(g for g, o in zip(given, ctx.outs) if o is not None and not o.requires_grad))
        return given if isinstance(outs, tuple) else given[0]

    @staticmethod
    def backward(ctx, *grads):
        outs, grads = zip(*((o, g) for o, g in zip(ctx.outs, grads) if g is not None))
        got = iter(torch.autograd.grad(outs, ctx.inputs, grads, retain_graph=True, allow_unused=True))
        return None, *(next(got) if grad else None for grad in ctx.needs_input_grad[1:])


def _traced(name: str, *args):
    """What a host operator calls in its place while a trace is recorded."""
    return _TracedStep.apply(getattr(host(), name), *args)


SIGS = {
    "pt_status_fetch_and_clear": "",
    "pt_sm_count": "",
    "pt_set_peer_wait_limit_ns": "L",
    "pt_gemm_bf16": "PPPIIIIIILLLLLLLLPIILIIIIIIPILP",
    "pt_gemm_bf16_kgroup2": "PPPLPPPLPIILLLLIIP",
    "pt_merge_partial": "PPPIPPIIIILP",
    "pt_rmsnorm_fwd": "PPPPPPIIFIP",
    "pt_rmsnorm_bwd_grid": "I",
    "pt_rmsnorm_bwd": "PPPPPPPIIIP",
    "pt_colsum_accumulate": "PIIIPIP",
    "pt_colsum_accumulate_pair": "PIIIPPIP",
    "pt_qk_norm_rope_fwd": "PPPPPPPPPPIIIIILFIP",
    "pt_qk_norm_rope_bwd_grid": "IIII",
    "pt_qk_norm_rope_bwd": "PPPPPPPPPPPPPIIIIILLIP",
    "pt_router_topk_fwd": "PIPPPIIIIIFP",
    "pt_router_given_fwd": "PIPPPIIIIFP",
    "pt_router_topk_bwd": "PPPPPPIIIIIIFP",
    "pt_route_sort": "PPIIIPLPPPIP",
    "pt_route_sort_noalloc": "PIIIPPPIP",
    "pt_gather_rows": "PPIPPIILP",
    "pt_embedding_bwd": "PPPIILP",
    "pt_indexed_bias_add": "PPPIPPIIP",
    "pt_segment_sum": "PIPPIPIP",
    "pt_combine": "PPPPPPIIIP",
    "pt_swiglu_fwd": "PPPIIIFFP",
    "pt_swiglu_bwd": "PPPPPPPIIIFFPP",
    "pt_cross_entropy": "PPPIILIP",
    "pt_scale_bf16": "PPLP",
    "pt_sumsq_grid": "",
    "pt_sumsq": "PILPP",
    "pt_adamw": "PIPIPPLPFFFFFFFP",
    "pt_muon_slabs": "LL",
    "pt_muon_momentum_sumsq": "PIPIPLLFPPP",
    "pt_frobenius_scales": "PIIPP",
    "pt_muon_orthogonalize": "PPPPPPIIIIPPIFFP",
    "pt_symm_malloc": "PL",
    "pt_symm_free": "P",
    "pt_ipc_export": "PP",
    "pt_ipc_import": "PP",
    "pt_ipc_close": "P",
    "pt_ipc_handle_size": "",
    "pt_can_access_peer": "II",
    "pt_symm_signal": "PIIIP",
    "pt_symm_wait": "PIIIP",
    "pt_symm_copy": "PPLIP",
    "pt_ep_chan_struct_size": "",
    "pt_ep_plan": "PIIIIIPPPPP",
    "pt_ep_push": "PIIPLPPPPPP",
    "pt_ep_receive": "PIIPPPPIP",
    "pt_ep_return": "PIIPPPPP",
    "pt_ep_wait_returned": "PIIP",
    "pt_ep_ack": "PIIP",
    "pt_axpby_bf16": "PPLFFP",
    "pt_fsdp_chan_struct_size": "",
    "pt_fsdp_ctl_bytes": "",
    "pt_fsdp_reduce_grid": "",
    "pt_fsdp_signal_ready": "PIP",
    "pt_fsdp_reduce_scatter": "PIFPP",
    "pt_fsdp_wait_acks": "PIP",
    "pt_fsdp_push_params": "PIP",
    "pt_fsdp_wait_params": "PIP",
    "pt_quant_rows": "PLPIPIIPPLP",
    "pt_quant_blocks": "PIIIPPPPP",
    "pt_gemm_fp8": "PPPIIIILLLLPLPPIIIIP",
    "pt_attn_fwd": "PPPPPPP" + "IIIIIII" + "LLLL" + "F" + "II" + "P",
    "pt_gated_attn_parts": "IIII",
    "pt_gated_attn_pre_fwd": "PPPPPPPPPIIIIILFP",
    "pt_gated_attn_pre_bwd": "PPPPPPPPPPPPIIIIILP",
    "pt_gated_attn_post_fwd": "PPLPIIIP",
    "pt_gated_attn_post_bwd": "PPPLPPIIIP",
    "pt_balanced_replay": "PIIIIP",
    "pt_packed_positions": "PIPLP",
    "pt_row_lower_bounds": "PIPIIIIP",
    "pt_attn_bwd_split": "PPPPPPPPPPPPP" + "IIIIIII" + "LLLLL" + "F" + "II" + "P",
    "pt_attn_bwd_split_reach": "PPPPPPPPPPPPP" + "IIIIIII" + "LLLLL" + "F" + "III" + "P",
    "pt_attn_bwd": "PPPPPPPPPPPPPPP" + "IIIIII" + "LLLLL" + "F" + "II" + "P",
    "pt_gemm2cta_nt": "PPPIIILLLP",
    "pt_dense_nn": "PPPIIILLLP",
    "pt_dense_tn": "PPPIIIIILLLP",
    "pt_mla_fwd": "PPPLLLPPPPPPIIIIIIIP",
    "pt_mla_bwd": "PPPPPPPPPIIIIIIIP",
    "pt_row_bias_dot": "PPPIPPPIIP",
    "pt_gdn_conv_fwd": "PPPPPIIIIP",
    "pt_gdn_conv_parts": "II",
    "pt_gdn_conv_bwd": "PPPPPPPIIIIP",
    "pt_gdn_gnorm_fwd": "PPPPLFP",
    "pt_gdn_gnorm_parts": "L",
    "pt_gdn_gnorm_bwd": "PPPPPPPLFP",
    "pt_gdr_fwd": "PPPPPPPPPPPPPP" + "III" + "F" + "P",
    "pt_gdr_bwd": "PPPPPPPPPPPPPPPPPPPP" + "III" + "F" + "P",
    "pt_gdr_state_fwd": "PPPPPPPPIIIIP",
    "pt_gdr_state_bwd": "PPPPPPPPPPPPPIIIIP",
}

_CT = {"P": c_void_p, "I": c_int, "L": c_longlong, "F": c_float}


def _declare(L: ctypes.CDLL) -> None:
    for name, args in SIGS.items():
        if hasattr(L, name):
            fn = getattr(L, name)
            fn.argtypes = [_CT[a] for a in args]
            fn.restype = c_int


def stream_ptr() -> int:
    """Handle of the current stream of the current device, without building a ``torch.cuda.Stream`` object: that took 17 us a
    call, a fifth of the host time of a launch-bound step."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def on_current_device(t: torch.Tensor) -> bool:
    """Whether launches of this module, which go to the current device, reach the memory of ``t``. Operations that take a kernel
    in place of tensor operations ask it, because those run on the device of their tensors."""
    return t.is_cuda and t.get_device() == torch._C._cuda_getDevice()


def ptr(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


_launches = 0
_LAUNCHES_PER_CALL = {"pt_attn_bwd": 3, "pt_gdr_fwd": 3, "pt_gdr_bwd": 3, "pt_merge_partial": 2}


def check(rc: int, what: str, launches: int | None = None) -> None:
    """Raise if ``rc`` is an error; ``launches``: the kernels that this call issued, where that depends on its arguments."""
    global _launches
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")
    _launches += _LAUNCHES_PER_CALL.get(what, 1) if launches is None else launches


def set_peer_wait_limit(seconds: float) -> None:
    """Limit of every in-kernel wait on another GPU's flag (current device). Bounded waits that run out set the status
    word, which the train step reads once per step; the default of 2 s suits tests, production jobs pass a longer one
    through ``DistributedCfg.peer_wait_timeout``."""
    rc = lib().pt_set_peer_wait_limit_ns(int(seconds * 1e9))
    if rc != 0:
        raise RuntimeError(f"pt_set_peer_wait_limit_ns failed with code {rc}")


def fetch_status() -> int:
    """Synchronise, read and clear the status word; returns the code (0 = no kernel reported anything)."""
    v = lib().pt_status_fetch_and_clear()
    if v < 0:
        raise RuntimeError(f"status word unavailable ({v})")
    return v


def check_status() -> None:
    """Synchronise and raise if any kernel recorded a timeout / overflow since the last check."""
    v = lib().pt_status_fetch_and_clear()
    if v > 0:
        raise KernelStatusError(STATUS_NAMES.get(v, f"status {v}"))
    if v < 0:
        raise RuntimeError(f"status word unavailable ({v})")


class _Module(types.ModuleType):
    """This module, with ``LAUNCHES``: kernels launched through it and through :func:`host` since it was last set to 0."""

    @property
    def LAUNCHES(self) -> int:
        return _launches + (host().launches() if host.cache_info().currsize else 0)

    @LAUNCHES.setter
    def LAUNCHES(self, value: int) -> None:
        global _launches
        _launches = value - (host().launches() if host.cache_info().currsize else 0)


sys.modules[__name__].__class__ = _Module
