"""Top-k softmax router: module, autograd function, functional entry point and the fp64 oracle.

Public surface of the reference's ``pkg/kernels/moe_router.py`` (``MoERouter``, ``MoERouterFunction`` /
``MoERouterAutograd``, ``moe_topk_route``, ``RouterProfile``, ``_reference_route_fp64``,
``_reference_backward_fp64``, ``_compute_load_imbalance``, ``_compute_router_z_loss``,
``_should_use_triton``, ``MIN_TRITON_DIM``, ``TRITON_AVAILABLE``).

On a CUDA device with bf16 tokens the whole forward is ONE sm_100a kernel (gate GEMM on tcgen05,
softmax, top-k, renormalisation, per-expert counts, load-balance sums, z-loss); the backward is one
elementwise kernel plus two tcgen05 GEMMs.  There is no Triton path (``TRITON_AVAILABLE`` is False and
``RouterProfile.used_triton`` is always False; ``used_fused_kernel`` says whether the sm_100a kernel ran).
Everywhere else (CPU, fp32 tokens, shapes the kernel does not cover) the fp64 PyTorch restatement runs;
it is also the test oracle.

Unlike the reference (``moe_router.py:690-734``) the module makes no host round trip per call: counts,
z-loss and the conservation check are produced on the device and only read when ``last_profile`` is.
The load-balance loss ``E * sum_i f_i * P_i`` and the z-loss are returned as differentiable tensors
(``last_aux_loss`` / ``last_z_loss``); the reference only had a non-differentiable z-loss float.
"""

from __future__ import annotations

import math
import os
from dataclasses import dataclass
from typing import Any, Dict, Optional, Tuple

import torch
import torch.nn as nn

from . import _ext, kernels

TRITON_AVAILABLE = False  # there is no Triton path in this package
MIN_TRITON_DIM = 16       # smallest N/H/E for which the reference dispatched its device kernel
MAX_FUSED_EXPERTS = 256
MAX_FUSED_TOPK = 8

__all__ = [
    "MoERouter",
    "MoERouterFunction",
    "MoERouterAutograd",
    "moe_topk_route",
    "RouterProfile",
    "TRITON_AVAILABLE",
]


# --------------------------------------------------------------------------------------------------
# fp64 oracle (also the CPU production path)
# --------------------------------------------------------------------------------------------------
def _reference_route_fp64(tokens: torch.Tensor, gate_w: torch.Tensor, k: int
                          ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """(topk_idx int64 [N,K], topk_w [N,K], logits [N,E]) computed in float64, cast back to the token dtype."""
    logits = tokens.to(torch.float64) @ gate_w.to(torch.float64)
    probs = torch.softmax(logits, dim=-1)
    vals, idx = torch.topk(probs, k=k, dim=-1, largest=True)
    w = vals / vals.sum(dim=-1, keepdim=True).clamp_min(1e-30)
    return idx.to(torch.long), w.to(tokens.dtype), logits.to(tokens.dtype)


def _reference_backward_fp64(logits: torch.Tensor, topk_idx: torch.Tensor, grad_w: torch.Tensor, k: int, E: int
                             ) -> torch.Tensor:
    """d(sum grad_w * w)/d(logits) in float64: through the renormalisation, the gather and the softmax."""
    probs = torch.softmax(logits.to(torch.float64), dim=-1)
    v = probs.gather(1, topk_idx)
    S = v.sum(dim=-1, keepdim=True).clamp_min(1e-30)
    gw = grad_w.to(torch.float64)
    grad_v = gw / S - (gw * v).sum(dim=-1, keepdim=True) / (S * S)
    grad_p = torch.zeros_like(probs).scatter_add_(1, topk_idx, grad_v)
    return probs * (grad_p - (grad_p * probs).sum(dim=-1, keepdim=True))


def _compute_load_imbalance(dispatch_cnt: torch.Tensor) -> float:
    cnt = dispatch_cnt.float()
    mean = float(cnt.mean())
    return 1.0 if mean < 1e-9 else float(cnt.max()) / mean


def _compute_router_z_loss(logits: torch.Tensor) -> float:
    return float((torch.logsumexp(logits.float(), dim=-1) ** 2).mean())


def _should_use_fused(tokens: torch.Tensor, gate_w: torch.Tensor, force_reference: bool, k: int = 1) -> bool:
    """Single source of truth for "will the sm_100a kernel run" (used for dispatch and for telemetry)."""
    if force_reference or not (tokens.is_cuda and gate_w.is_cuda):
        return False
    if os.environ.get("CMOE_FORCE_LIBRARY", "0") == "1":  # the benchmarks' library arm: no device code of this package
        return False
    if tokens.dtype != torch.bfloat16 or tokens.dim() != 2:
        return False
    N, H = tokens.shape
    E = gate_w.shape[1]
    return (N >= 1 and H % 8 == 0 and E % 8 == 0 and E <= MAX_FUSED_EXPERTS and 1 <= k <= min(MAX_FUSED_TOPK, E)
            and tokens.stride(1) == 1 and (tokens.stride(0) * 2) % 16 == 0)


def _next_pow2(n: int) -> int:
    """Smallest power of two >= n (the reference sizes its expert tile with it, moe_router.py:297-388; the fused
    kernel pads the expert dimension to a multiple of 16 instead, this stays for callers of the helper)."""
    return 1 if n <= 1 else 1 << (int(n) - 1).bit_length()


def _should_use_triton(tokens: torch.Tensor, gate_w: torch.Tensor, force_reference: bool) -> bool:
    """Kept for callers of the reference API: true when a device kernel (here: the fused sm_100a one) runs."""
    return _should_use_fused(tokens, gate_w, force_reference)


# --------------------------------------------------------------------------------------------------
# fused device path
# --------------------------------------------------------------------------------------------------
class RouterOutput:
    """Everything the fused forward produced, all on the device.  ``idx32`` / ``w32`` are what the kernels downstream
    read, ``idx64`` / ``w16`` / ``counts64`` the same values in the types that the public entry points return."""

    __slots__ = ("idx32", "w32", "idx64", "w16", "logits", "lse", "counts", "counts64", "mean_prob", "stats", "events")

    def __init__(self, idx32, w32, idx64, w16, logits, lse, counts, counts64, mean_prob, stats, events=None):
        self.idx32, self.w32, self.idx64, self.w16 = idx32, w32, idx64, w16
        self.logits, self.lse, self.counts, self.counts64 = logits, lse, counts, counts64
        self.mean_prob, self.stats, self.events = mean_prob, stats, events


def fused_router_forward(tokens: torch.Tensor, gate_w_bf16: torch.Tensor, k: int, timed: bool = False) -> RouterOutput:
    ext, status = _ext.ext(), kernels.status_word(tokens.device)
    if not timed:
        return RouterOutput(*ext.router_route(tokens, gate_w_bf16, k, True, status))
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    out = RouterOutput(*ext.router_route(tokens, gate_w_bf16, k, True, status), events=(e0, e1))
    e1.record()
    return out


def _bf16_gate(gate_w: torch.Tensor) -> torch.Tensor:
    return (gate_w if gate_w.dtype == torch.bfloat16 else gate_w.to(torch.bfloat16)).contiguous()


def _fused_router_backward(ctx, tokens, gw16, logits, lse, idx32, counts, grad_w32, grad_w16, grad_aux, grad_z,
                           gate_dtype):
    """(grad_tokens, grad_gate): the analytic d(logits) kernel and the two contractions with it."""
    gt, gg = _ext.ext().router_grad(tokens, gw16, logits, lse, idx32, counts, grad_w32, grad_w16, grad_aux, grad_z,
                                    ctx.needs_input_grad[0], ctx.needs_input_grad[1], gate_dtype == torch.bfloat16,
                                    kernels.status_word(tokens.device))
    return gt, (gg if gg is None or gg.dtype == gate_dtype else gg.to(gate_dtype))


class FusedRouterFunction(torch.autograd.Function):
    """(tokens, gate_w) -> (gate weights fp32, gate weights in bf16 [N,K], aux loss, z loss, idx32, idx64); the two
    weight tensors hold the same values and take gradients each.  Everything else rides on ``holder``."""

    @staticmethod
    def forward(ctx, tokens, gate_w, k: int, holder: Dict[str, Any], timed: bool):
        gw16 = _bf16_gate(gate_w)
        out = fused_router_forward(tokens, gw16, k, timed)
        holder["out"] = out
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(tokens, gw16, out.logits, out.lse, out.idx32, out.counts)
        ctx.gate_dtype = gate_w.dtype
        ctx.mark_non_differentiable(out.idx32, out.idx64)
        return out.w32, out.w16, out.stats[0], out.stats[1], out.idx32, out.idx64

    @staticmethod
    def backward(ctx, grad_w32, grad_w16, grad_aux, grad_z, _grad_idx32, _grad_idx64):
        gt, gg = _fused_router_backward(ctx, *ctx.saved_tensors, grad_w32, grad_w16, grad_aux, grad_z, ctx.gate_dtype)
        return gt, gg, None, None, None


# --------------------------------------------------------------------------------------------------
# autograd function with the reference's signature
# --------------------------------------------------------------------------------------------------
class MoERouterFunction(torch.autograd.Function):
    """``apply(tokens[N,H], gate_w[H,E], k, force_reference=False, report=None) -> (idx int64, w)``."""

    @staticmethod
    def forward(ctx, tokens, gate_w, k: int, force_reference: bool = False, report: Optional[dict] = None):
        N, H = tokens.shape
        E = gate_w.shape[1]
        fused = _should_use_fused(tokens, gate_w, force_reference, k)
        if fused:
            gw16 = _bf16_gate(gate_w)
            out = fused_router_forward(tokens, gw16, k, timed=report is not None)
            idx, w, logits = out.idx64, out.w16, out.logits
            ctx.fused_saved = (gw16, out.lse, out.idx32, out.counts)
            if report is not None:
                report["output"] = out
        else:
            idx, w, logits = _reference_route_fp64(tokens, gate_w, k)
            ctx.fused_saved = None
        if report is not None:
            report["used_fused_kernel"] = fused
            report["used_triton"] = False
            report["logits"] = logits
        ctx.save_for_backward(tokens, gate_w, logits, idx)
        ctx.k, ctx.E, ctx.fused = k, E, fused
        ctx.mark_non_differentiable(idx)
        return idx, w

    @staticmethod
    def backward(ctx, _grad_idx, grad_w):
        tokens, gate_w, logits, idx = ctx.saved_tensors
        if ctx.fused:
            gw16, lse, idx32, counts = ctx.fused_saved
            gt, gg = _fused_router_backward(ctx, tokens, gw16, logits, lse, idx32, counts, None, grad_w, None, None,
                                            gate_w.dtype)
            return gt, gg, None, None, None
        gl = _reference_backward_fp64(logits, idx, grad_w, ctx.k, ctx.E)
        grad_tokens = (gl @ gate_w.to(torch.float64).t()).to(tokens.dtype) if ctx.needs_input_grad[0] else None
        grad_gate = (tokens.to(torch.float64).t() @ gl).to(gate_w.dtype) if ctx.needs_input_grad[1] else None
        return grad_tokens, grad_gate, None, None, None


MoERouterAutograd = MoERouterFunction


def moe_topk_route(tokens: torch.Tensor, gate_w: torch.Tensor, k: int, force_reference: bool = False
                   ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Route ``[B,S,H]`` or ``[N,H]`` tokens; returns ``(idx int64 [N,K], w [N,K])``."""
    if tokens.dim() == 3:
        tokens = tokens.reshape(-1, tokens.shape[-1])
    elif tokens.dim() != 2:
        raise ValueError(f"tokens must be [B,S,H] or [N,H], got shape {list(tokens.shape)}")
    if not (1 <= k <= gate_w.shape[1]):
        raise ValueError(f"k={k} must be in [1, {gate_w.shape[1]}]")
    if not kernels.needs_autograd(tokens, gate_w) and _should_use_fused(tokens, gate_w, force_reference, k):
        # no gradient wanted: one native call, one kernel, and only the decision itself is written
        out = _ext.ext().router_route(tokens, _bf16_gate(gate_w), k, False, kernels.status_word(tokens.device))
        return out[2], out[3]
    return MoERouterFunction.apply(tokens, gate_w, k, force_reference, None)


# --------------------------------------------------------------------------------------------------
# module
# --------------------------------------------------------------------------------------------------
def _fused_stage_bytes(num_experts: int) -> int:
    """Shared memory of one 64-wide k-block of a full 128-token tile of the fused router kernel (csrc/router.cu): the
    bf16 slice of the activations plus the matching slice of the gate weights, experts padded to a multiple of 64.  (A
    pipeline stage holds two k-blocks; few tokens get shorter tiles, and wide gates are split over a cluster.)
    Reported on every path as the on-chip working set per block, like the reference's theoretical figure
    (pkg/kernels/moe_router.py:703-714)."""
    e_chunks = max(1, (num_experts + 63) // 64)
    return 128 * 64 * 2 + e_chunks * 64 * 64 * 2


@dataclass
class RouterProfile:
    sram_bytes_per_block: int = 0
    achieved_bandwidth_gbps: float = 0.0
    kernel_ms: float = 0.0
    used_triton: bool = False
    tokens_per_expert_mean: float = 0.0
    tokens_per_expert_std: float = 0.0
    expert_load_imbalance: float = 1.0
    router_z_loss: float = 0.0
    used_fused_kernel: bool = False
    backend: str = "torch-fp64"
    aux_loss: float = 0.0
    dispatch_counts: Optional[list] = None


class MoERouter(nn.Module):
    """Learned top-k router.  ``forward(tokens[N,H]) -> (idx int64 [N,K], w [N,K], dispatch_cnt int64 [E])``."""

    def __init__(self, hidden_dim: int, num_experts: int, top_k: int = 2, bias: bool = False,
                 dtype: torch.dtype = torch.float32):
        super().__init__()
        if not (1 <= top_k <= num_experts):
            raise ValueError(f"top_k={top_k} must be in [1, num_experts={num_experts}]")
        self.hidden_dim, self.num_experts, self.top_k = hidden_dim, num_experts, top_k
        self.gate_w = nn.Parameter(torch.empty(hidden_dim, num_experts, dtype=dtype))
        nn.init.normal_(self.gate_w, mean=0.0, std=1.0 / math.sqrt(hidden_dim))
        self.bias = nn.Parameter(torch.zeros(num_experts, dtype=dtype)) if bias else None
        self.profile_timing = False  # record CUDA events around the kernel (resolved lazily)
        self._pending: Optional[dict] = None
        self._profile: Optional[RouterProfile] = None
        self._last_logits: Optional[torch.Tensor] = None
        self.last_aux_loss: Optional[torch.Tensor] = None
        self.last_z_loss: Optional[torch.Tensor] = None
        self.last_idx32: Optional[torch.Tensor] = None
        self.last_w32: Optional[torch.Tensor] = None

    def extra_repr(self) -> str:
        return f"hidden_dim={self.hidden_dim}, num_experts={self.num_experts}, top_k={self.top_k}"

    # the statistics of the last call are materialised (one device read) only when somebody asks
    @property
    def last_profile(self) -> Optional[RouterProfile]:
        if self._pending is not None:
            self._profile = self._materialise(self._pending)
            self._pending = None
        return self._profile

    @last_profile.setter
    def last_profile(self, value: Optional[RouterProfile]) -> None:
        self._pending, self._profile = None, value

    def _materialise(self, pend: dict) -> RouterProfile:
        counts = pend["counts"].detach().to("cpu", torch.float64)
        N, H, E, K = pend["N"], self.hidden_dim, self.num_experts, self.top_k
        total = int(counts.sum())
        if total != N * K:
            raise RuntimeError(
                f"Token conservation violation: dispatched {total} (token, slot) pairs, expected {N * K} "
                f"(N={N}, K={K})")
        kernel_ms = 0.0
        if pend.get("events") is not None:
            e0, e1 = pend["events"]
            e1.synchronize()
            kernel_ms = e0.elapsed_time(e1)
        bytes_moved = N * H * pend["elem"] + H * E * pend["elem"] + N * E * 4 + N * K * 8
        if pend.get("stats") is not None:  # the fused kernel's {aux loss, z loss, ...}
            aux, z = pend["stats"].tolist()[:2]
        else:
            aux, z = float(pend["aux_loss"]), float(pend["z_loss"])
        mean = float(counts.mean())
        return RouterProfile(
            sram_bytes_per_block=_fused_stage_bytes(E),
            achieved_bandwidth_gbps=(bytes_moved / (kernel_ms * 1e6)) if kernel_ms > 0 else 0.0,
            kernel_ms=kernel_ms,
            used_triton=False,
            tokens_per_expert_mean=mean,
            tokens_per_expert_std=float(counts.std(unbiased=False)) if E > 1 else 0.0,
            expert_load_imbalance=(float(counts.max()) / mean) if mean > 1e-9 else 1.0,
            router_z_loss=z,
            used_fused_kernel=pend["fused"],
            backend="sm100a-fused" if pend["fused"] else "torch-fp64",
            aux_loss=aux,
            dispatch_counts=[int(c) for c in counts.tolist()],
        )

    def forward(self, tokens: torch.Tensor, force_reference: bool = False
                ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
        if tokens.dim() == 3:
            tokens = tokens.reshape(-1, tokens.shape[-1])
        if tokens.dim() != 2 or tokens.shape[1] != self.hidden_dim:
            raise ValueError(f"expected tokens [N, {self.hidden_dim}], got {list(tokens.shape)}")
        N = tokens.shape[0]
        E, K = self.num_experts, self.top_k
        fused = self.bias is None and _should_use_fused(tokens, self.gate_w, force_reference, K)
        if fused:
            if not kernels.needs_autograd(tokens, self.gate_w):
                out = fused_router_forward(tokens, _bf16_gate(self.gate_w), K, self.profile_timing)
                w32, w, idx32, idx = out.w32, out.w16, out.idx32, out.idx64
                aux, z = out.stats[0], out.stats[1]
            elif (tokens.is_cuda and self.gate_w.dtype == torch.bfloat16 and self.gate_w.is_contiguous()
                  and not self.profile_timing and not kernels.traced_or_dual(tokens, self.gate_w)):
                fields, aux, z = _ext.ext().router_node(tokens, self.gate_w, K, kernels.status_word(tokens.device))
                out = RouterOutput(*fields)
                w32, w, idx32, idx = out.w32, out.w16, out.idx32, out.idx64
            else:
                holder: Dict[str, Any] = {}
                w32, w, aux, z, idx32, idx = FusedRouterFunction.apply(tokens, self.gate_w, K, holder,
                                                                       self.profile_timing)
                out: RouterOutput = holder["out"]
            left = dict(_last_logits=out.logits, last_aux_loss=aux, last_z_loss=z, last_idx32=idx32, last_w32=w32,
                        _pending=dict(counts=out.counts, N=N, fused=True, events=out.events, stats=out.stats, elem=2))
            if type(self) is MoERouter:
                # plain attributes of this class, set past the module's look at each for parameters and buffers
                self.__dict__.update(left)
            else:
                for name, value in left.items():
                    setattr(self, name, value)
            return idx, w, out.counts64
        # PyTorch path (bias, CPU, fp32 tokens, shapes the kernel does not cover): fp64 math under autograd
        logits64 = tokens.to(torch.float64) @ self.gate_w.to(torch.float64)
        if self.bias is not None:
            logits64 = logits64 + self.bias.to(torch.float64)
        probs = torch.softmax(logits64, dim=-1)
        vals, idx = torch.topk(probs, K, dim=-1, largest=True)
        w = (vals / vals.sum(-1, keepdim=True).clamp_min(1e-30)).to(tokens.dtype)
        counts = torch.bincount(idx.reshape(-1), minlength=E)
        f = counts.to(torch.float64) / float(N * K)
        self.last_aux_loss = (E * (f * probs.mean(0)).sum()).to(torch.float32)
        self.last_z_loss = (torch.logsumexp(logits64, dim=-1) ** 2).mean().to(torch.float32)
        self._last_logits = logits64.detach().to(tokens.dtype)
        self.last_idx32, self.last_w32 = idx.to(torch.int32), w.float()
        self._pending = dict(counts=counts, N=N, fused=False, events=None, z_loss=self.last_z_loss.detach(),
                             aux_loss=self.last_aux_loss.detach(), elem=tokens.element_size())
        return idx, w, counts
