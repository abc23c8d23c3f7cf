"""Host side of the B200 gated scan: the reference's scan interface over the C ABI.

Mirrors naju/scan.py of the reference project: the same `naju_scan` signature
(naju/scan.py:75-76), the same tensor meaning (naju/scan.py:3-12) and the same backend
selection rule (argument > NAJU_SCAN_BACKEND > default, naju/scan.py:48-52).  There is one
implementation behind it — hand-written sm_100a CUDA in libnaju_b200.so — and no fallback:
a CPU tensor or a missing library raises.

Additive, keyword-only extensions the reference does not have: an initial state `h0`, the
returned final state, and `naju_scan_step` for single-token decode.
"""
import os

import torch

from . import _lib
from ._lib import native as _native

# The reference's backend names are accepted so that existing configs keep working
# (naju/mixer.py:121-122 forwards `scan_backend`); they all select the one CUDA path.
_ALIASES = ("b200", "reference", "chunk", "cuda", "cuda_bw", "affine", "fused_affine_chunk")

def resolve_backend(backend=None):
    """Same precedence as naju/scan.py:48-52; every valid name resolves to "b200"."""
    b = backend or os.environ.get("NAJU_SCAN_BACKEND") or "b200"
    b = b.lower()
    if b not in _ALIASES:
        raise ValueError(f"unknown scan backend {b!r}; valid: {', '.join(_ALIASES)}")
    return "b200"


# Switches read by every call (naju_b200/csrc/torch_host.cpp):
#   NAJU_B200_FORM selects the kernel family: "auto" (default) takes the tcgen05 tensor-core chunked form
#   where it applies (16-bit activations, bf16 B/C, TMA-legal strides, N == 16 -- or fewer, padded with zero
#   columns by the host when the problem is large enough --; bf16 activations and 17 to 64 states where there are
#   channel tiles enough) and the exact recurrent kernels elsewhere; "recurrent" forces the recurrent ones;
#   "chunked" insists on the 16-state tensor-core form and raises where it does not apply.
#   NAJU_B200_CHECK_STATUS=1 reads the device-side status word after every call (synchronises the stream).
#   NAJU_B200_INJECT_TIMEOUT=1 is the fault injection for tests, NAJU_B200_GUARD=1 the canary bands below.


def last_kernel_forms():
    """{"fwd": form, "bwd": form}: the kernel family (FORM_* of _lib) that did the work of the most recent
    calls made with NAJU_B200_CHECK_STATUS=1 (None before the first)."""
    f, b = _native().forms()
    return {"fwd": None if f < 0 else f, "bwd": None if b < 0 else b}


def _time_contig(u):
    """True for a [B,T,D] view of [B,D,T] memory (time stride 1, channels T or more apart) that
    the kernels can take as it is: what the mixer's depthwise convolution leaves behind
    (naju/mixer.py:115).  TMA wants the channel and batch strides to be multiples of 16 bytes."""
    return _native().time_contig(u)


def _prepare(u, f_logit, i_logit, Bm, Cm, D_skip):
    """The six inputs as the kernels take them: checked, logits in u's dtype or fp32, B and C in their
    common dtype or fp32, D_skip fp32; copied only where a layout cannot be described."""
    return _native().prepare(u, f_logit, i_logit, Bm, Cm, D_skip)


def _desc(u, f_logit, i_logit, Bm, Cm):
    """The C ABI's descriptor of prepared inputs (struct naju_scan_desc)."""
    return _lib.ScanDesc.from_buffer_copy(_native().describe(u, f_logit, i_logit, Bm, Cm))


# With NAJU_B200_GUARD=1 every workspace sits between two canary bands of _GUARD bytes that
# check_workspace_guards() verifies: the stand-in for a memory checker on the kernels' writes to
# checkpoint and scratch buffers (a debug aid; off by default).
_GUARD = 4096
_GUARD_BYTE = 0xA5


def check_workspace_guards():
    """Verifies (and forgets) the canary bands of every workspace handed out under
    NAJU_B200_GUARD=1 since the last call; raises if a kernel wrote outside its workspace.
    Synchronises the device."""
    guarded = _native().take_guarded()
    bad = []
    for whole, n in guarded:
        lo, hi = whole[:_GUARD], whole[_GUARD + n:]
        if bool((lo != _GUARD_BYTE).any()) or bool((hi != _GUARD_BYTE).any()):
            bad.append((int(whole.numel()), n))
    if bad:
        raise RuntimeError(f"workspace guard bands overwritten: {bad}")
    return len(guarded)


def _state_arg(h, B, D, N, name):
    return _native().state_arg(h, B, D, N, name)


# (N < 16 on a large 16-bit problem is padded with zero columns to the 16 states of the tcgen05 kernels.
# The same argument splits N > 16 into groups of 16 states whose y / du / d f_logit / d i_logit are added
# up; that was built and measured, but every group's output is rounded to the 16-bit activation type before
# the sum, which put y and the gradients at 2.7e-3 of the reference, outside the 1e-3 / 2e-3 bounds: 17 to 64
# states have kernels of their own.)
_GROUP = 16


def scan_forward(u, f_logit, i_logit, Bm, Cm, D_skip, h0=None, want_final=False, want_decay=False):
    """Raw forward over prepared tensors.  Returns (y, hT|None, pT|None, ckpt, desc)."""
    y, hT, pT, ckpt, desc = _native().forward(u, f_logit, i_logit, Bm, Cm, D_skip, h0, want_final, want_decay)
    return y, hT, pT, ckpt, _lib.ScanDesc.from_buffer_copy(desc)


def scan_backward(d, u, f_logit, i_logit, Bm, Cm, D_skip, h0, dy, dhT, ckpt, want_dh0=False):
    """Raw backward.  Returns (du, dfl, dil, dB, dC, dD, dh0|None).  `d` and `ckpt` are what
    scan_forward returned for the same tensors (NAJU_B200_FORM must not change in between: it
    decides whether fewer than 16 states are padded)."""
    return _native().backward(d.flags, u, f_logit, i_logit, Bm, Cm, D_skip, h0, dy, dhT, ckpt, want_dh0)


# ---------------------------------------------------------------------------------------------
# The same forward / backward as torch.library custom ops, so that torch.compile does not break
# the graph at the scan (the reference's scan is a graph break: naju/README.md:99-100) and
# NajuBlock(use_ckpt=True) (naju/mixer.py:139-141) composes.  Used while compiling; eager calls
# go to the native autograd node (naju_b200/csrc/torch_host.cpp).
def _ckpt_bytes_formula(B, T, D, N, act, bdt):
    """Size of the checkpoint buffer (naju_b200_ckpt_bytes) as arithmetic that also works on the
    symbolic sizes of fake tensors."""
    NS = 16 if N <= 16 else 32 if N <= 32 else 64 if N <= 64 else 128
    TC = 64 if (N == 16 and act in (torch.bfloat16, torch.float16) and bdt == torch.bfloat16 and D % 8 == 0) else 32
    ntiles = ((T + TC - 1) // TC) * B * ((D + 127) // 128)
    a256 = lambda x: (x + 255) // 256 * 256
    return a256(ntiles * 128 * NS * 4) + a256(ntiles * 128 * 4) + 256


def _pads_to_group(work, T, N, act, bdt):
    """The host's padding rule for fewer than 16 states (pad_to_group of torch_host.cpp) as arithmetic on
    the symbolic sizes of fake tensors."""
    if N >= _GROUP or os.environ.get("NAJU_B200_FORM", "auto").lower() == "recurrent":
        return False
    return act in (torch.bfloat16, torch.float16) and bdt == torch.bfloat16 and work >= 1 << 20 and T >= 128


@torch.library.custom_op("naju_b200::scan_fwd", mutates_args=())
def _scan_fwd_op(u: torch.Tensor, f_logit: torch.Tensor, i_logit: torch.Tensor, Bm: torch.Tensor,
                 Cm: torch.Tensor, D_skip: torch.Tensor, h0: torch.Tensor,
                 want_final: bool) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    pu, pf, pi, pB, pC, pD = _prepare(u, f_logit, i_logit, Bm, Cm, D_skip)
    B, T, D = pu.shape
    ph0 = _state_arg(h0, B, D, pB.shape[-1], "h0") if h0.numel() else None
    y, hT, _, ckpt, _ = scan_forward(pu, pf, pi, pB, pC, pD, ph0, want_final=want_final)
    return y, (hT if want_final else y.new_empty(0, dtype=torch.float32)), ckpt


@_scan_fwd_op.register_fake
def _(u, f_logit, i_logit, Bm, Cm, D_skip, h0, want_final):
    B, T, D = u.shape
    N = Bm.shape[-1]
    hT = u.new_empty((B, D, N), dtype=torch.float32) if want_final else u.new_empty(0, dtype=torch.float32)
    # (fewer than 16 states may be padded to 16: the same rule as scan_forward, on the dtype
    # the prepared B and C take, see _prepare)
    bdt = Bm.dtype if Bm.dtype == Cm.dtype else torch.float32
    if _pads_to_group(B * T * D, T, N, u.dtype, bdt):
        N = _GROUP
    ckpt = u.new_empty(_ckpt_bytes_formula(B, T, D, N, u.dtype, bdt), dtype=torch.uint8)
    return u.new_empty((B, T, D)), hT, ckpt


@torch.library.custom_op("naju_b200::scan_bwd", mutates_args=())
def _scan_bwd_op(u: torch.Tensor, f_logit: torch.Tensor, i_logit: torch.Tensor, Bm: torch.Tensor,
                 Cm: torch.Tensor, D_skip: torch.Tensor, h0: torch.Tensor, dy: torch.Tensor,
                 dhT: torch.Tensor, ckpt: torch.Tensor) -> list[torch.Tensor]:
    pu, pf, pi, pB, pC, pD = _prepare(u, f_logit, i_logit, Bm, Cm, D_skip)
    B, T, D = pu.shape
    N = pB.shape[-1]
    ph0 = _state_arg(h0, B, D, N, "h0") if h0.numel() else None
    pdhT = _state_arg(dhT, B, D, N, "dhT") if dhT.numel() else None
    d = _desc(pu, pf, pi, pB, pC)
    du, dfl, dil, dB, dC, dD, dh0 = scan_backward(d, pu, pf, pi, pB, pC, pD, ph0, dy, pdhT, ckpt,
                                                  want_dh0=ph0 is not None)
    if dh0 is None:
        dh0 = du.new_empty(0, dtype=torch.float32)
    # (the fake implementation promises contiguous gradients: a du that came back in the layout of a
    # time-contiguous u is made contiguous here)
    return [du.to(u.dtype).contiguous(), dfl.to(f_logit.dtype), dil.to(i_logit.dtype), dB.to(Bm.dtype), dC.to(Cm.dtype),
            dD.to(D_skip.dtype), dh0.to(h0.dtype)]


@_scan_bwd_op.register_fake
def _(u, f_logit, i_logit, Bm, Cm, D_skip, h0, dy, dhT, ckpt):
    return [torch.empty_like(u, memory_format=torch.contiguous_format),
            torch.empty_like(f_logit, memory_format=torch.contiguous_format),
            torch.empty_like(i_logit, memory_format=torch.contiguous_format),
            torch.empty_like(Bm, memory_format=torch.contiguous_format),
            torch.empty_like(Cm, memory_format=torch.contiguous_format),
            torch.empty_like(D_skip), torch.empty_like(h0)]


def _scan_op_setup(ctx, inputs, output):
    u, f_logit, i_logit, Bm, Cm, D_skip, h0, want_final = inputs
    ctx.save_for_backward(u, f_logit, i_logit, Bm, Cm, D_skip, h0, output[2])
    ctx.want_final = want_final


def _scan_op_backward(ctx, dy, dhT, _dckpt):
    u, f_logit, i_logit, Bm, Cm, D_skip, h0, ckpt = ctx.saved_tensors
    if dy is None:
        dy = torch.zeros_like(u)
    if dhT is None or not ctx.want_final:
        dhT = u.new_empty(0, dtype=torch.float32)
    du, dfl, dil, dB, dC, dD, dh0 = _scan_bwd_op(u, f_logit, i_logit, Bm, Cm, D_skip, h0, dy.contiguous(),
                                                 dhT, ckpt)
    return du, dfl, dil, dB, dC, dD, (dh0 if h0.numel() else None), None


_scan_fwd_op.register_autograd(_scan_op_backward, setup_context=_scan_op_setup)


def _scan_via_custom_op(u, f_logit, i_logit, B, C, D_skip, h0, want_final):
    h0t = h0 if h0 is not None else u.new_empty(0, dtype=torch.float32)
    y, hT, _ = _scan_fwd_op(u, f_logit, i_logit, B, C, D_skip, h0t, want_final)
    return (y, hT) if want_final else y


def _by_custom_op():
    """Whether a compiler or a tracer is looking: it then has to find one op (what the native function does inside would be
    recorded as the allocation of its outputs and nothing else)."""
    return torch.compiler.is_compiling() or torch.jit.is_tracing()


def naju_b200_scan(u, f_logit, i_logit, B, C, D_skip):
    """Backend callable with the reference's 6-tensor signature (naju/scan.py:3-5)."""
    if _by_custom_op():
        return _scan_via_custom_op(u, f_logit, i_logit, B, C, D_skip, None, False)
    return _native().scan(u, f_logit, i_logit, B, C, D_skip, None, False)


def naju_scan(u, f_logit, i_logit, B, C, D_skip, backend=None, *, h0=None,
              return_final_state=False):
    """y = scan(u, f_logit, i_logit, B, C, D_skip) — drop-in for naju/scan.py:75-76.

    u, f_logit, i_logit [B,T,D]; B, C [B,T,N]; D_skip [D]; y [B,T,D] in u's dtype.
    Differentiable w.r.t. all six tensors (and h0).  With return_final_state=True returns
    (y, hT) where hT [B,D,N] fp32 is the state after the last step.
    """
    resolve_backend(backend)
    if _by_custom_op():
        return _scan_via_custom_op(u, f_logit, i_logit, B, C, D_skip, h0, bool(return_final_state))
    return _native().scan(u, f_logit, i_logit, B, C, D_skip, h0, return_final_state)


def naju_scan_step(state, u_t, f_logit_t, i_logit_t, B_t, C_t, D_skip):
    """Single-token decode update: one iteration of naju/scan.py:87-91.

    state [B,D,N] fp32 (updated IN PLACE); u_t, f_logit_t, i_logit_t [B,D]; B_t, C_t [B,N].
    Returns (y_t [B,D] in u_t's dtype, state).
    """
    return _native().step(state, u_t, f_logit_t, i_logit_t, B_t, C_t, D_skip)
