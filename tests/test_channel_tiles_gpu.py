"""16 states with few channel tiles (batch rows x 128 channels): which kernels take such a problem, and thread-block clusters that
share a channel tile, against the fp64 oracle."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

TICKET, WALK, RECURRENT = 2, 3, 1
BF, F32 = torch.bfloat16, torch.float32


@pytest.fixture(autouse=True)
def _status_checks(monkeypatch):
    monkeypatch.setenv("NAJU_B200_CHECK_STATUS", "1")


def _round(x, dt):
    return torch.tensor(x).to(dt).float().numpy()


def _run(B, T, D, f_shift, gdt, utm, states=True, f_logit=None, N=16):
    """((y, hT, gradients, forms), the oracle's)"""
    from naju_b200 import naju_scan
    from naju_b200.scan import last_kernel_forms
    d = oracle.make_inputs(B, T, D, N, seed=21, f_shift=f_shift, d_skip_scale=0.05, with_h0=True)
    if f_logit is not None:
        f_logit(d["fl"])
    cast = {"u": BF, "Bm": BF, "Cm": BF, "dy": BF, "fl": gdt, "il": gdt}
    q = {k: (_round(d[k], cast[k]) if k in cast else d[k]) for k in d}
    t = {k: torch.tensor(q[k], device="cuda").to(cast.get(k, F32)) for k in q}
    if utm:
        t["u"] = t["u"].transpose(1, 2).contiguous().transpose(1, 2)
    order = ("u", "fl", "il", "Bm", "Cm", "Dskip")
    x = {k: t[k].requires_grad_(True) for k in order + ("h0",)}
    y, hT = naju_scan(*(x[k] for k in order), h0=x["h0"] if states else None, return_final_state=True)
    torch.autograd.backward([y, hT], [t["dy"], t["dhT"] if states else torch.zeros_like(hT)])
    torch.cuda.synchronize()
    forms = last_kernel_forms()
    a, h0, dhT = [q[k] for k in order], (q["h0"] if states else None), (q["dhT"] if states else None)
    yo, hTo = oracle.oracle_fwd(*a, h0=h0, return_final_state=True)
    go = oracle.oracle_bwd(*a, q["dy"], h0=h0, dhT=dhT)
    g = {"du": x["u"].grad, "dfl": x["fl"].grad, "dil": x["il"].grad, "dB": x["Bm"].grad, "dC": x["Cm"].grad, "dD": x["Dskip"].grad}
    if states:
        g["dh0"] = x["h0"].grad
    return (y.detach(), hT.detach(), g, forms), (yo, hTo, go)


def _err(ours, want):
    return oracle.rel_l2(ours.double().cpu().numpy(), _round(want, BF) if ours.dtype == BF else want)


# B, T, D, f_shift, logits, time-contiguous u, initial state and its gradient
@pytest.mark.parametrize("case", [
    (8, 128, 2048, 5.0, F32, False, False),   # enough channel tiles, two chunks
    (8, 192, 2048, 2.0, BF, False, True),     # three
    (3, 509, 1536, 5.0, F32, False, True),    # 36 channel tiles
    (3, 509, 1536, 2.0, BF, False, False),
    (2, 520, 1024, 2.0, F32, True, True)])
def test_gradients_of_few_channel_tiles_or_chunks_are_fp32_inside(case):
    """The tensor-core backward's operands have 16 bits; problems that it need not take keep the recurrent kernel's fp32: dh0, dD and the
    gradient of fp32 write logits to 2e-6 (1e-5 and 3e-5 otherwise).  The states come from the forward's checkpoints, whose
    tensor-core kernel leaves 1e-5 in them: that is what the gradient of fp32 retention logits may show (2e-5 and 6e-5
    otherwise), and what moves 16-bit gradients: an error e before rounding to steps s moves e / s of the values by a step, sqrt(e s)
    in the 2-norm, 2.3e-4 for 1e-5 and s = 2^-7.5."""
    B, T, D, fs, gdt, utm, states = case
    (_, _, g, forms), (_, _, go) = _run(B, T, D, fs, gdt, utm, states)
    assert forms["bwd"] == RECURRENT
    for k in g:
        assert _err(g[k], go[k]) < (2.5e-4 if g[k].dtype == BF else 1e-5 if k == "dfl" else 2e-6), k


# B, T, D, f_shift, logits
@pytest.mark.parametrize("case", [(1, 1024, 2048, 5.0, F32), (2, 520, 1024, 2.0, BF), (8, 192, 2048, 2.0, F32)])
def test_time_contiguous_u_with_few_channel_tiles_keeps_an_fp32_state(case):
    """The recurrent kernel: final state to 2e-6 (1e-5 with the tensor-core kernel's operands of 16 bits), y a step apart in one place
    of 2000 at most (sqrt(1e-6 2^-7.5) = 7e-5)."""
    B, T, D, fs, gdt = case
    (y, hT, _, forms), (yo, hTo, _) = _run(B, T, D, fs, gdt, True)
    assert forms["fwd"] == RECURRENT
    assert _err(hT, hTo) < 2e-6
    assert _err(y, yo) < 7e-5


def _deep(chunks, channels):
    """Retention gates of some chunks and channels so deep that the chunk's product leaves fp32."""
    def change(fl):
        for c in chunks:
            fl[:, 64 * c + 5: 64 * c + 60, channels] = -9.0
    return change


# B, T, D, f_shift, logits, time-contiguous u, initial state, chunks with deep gates
@pytest.mark.parametrize("case", [
    # clusters of two: 38 and 40 channel tiles (the last of 8 channels), nine chunks (the last of 8 steps)
    (2, 520, 2432, 2.0, BF, False, True, ()),
    (2, 520, 2440, 2.0, F32, False, True, ()),
    (2, 520, 2440, 4.0, BF, True, True, ()),
    (2, 520, 2432, 2.0, F32, True, False, ()),
    (2, 520, 2432, 2.0, BF, False, True, (3,)),          # a deep tile between two mails
    (2, 520, 2440, 2.0, F32, True, True, (0, 1, 8)),     # ... the first two and the last
    # clusters of four (forward): 24 and 27 channel tiles, seven chunks; three, so that one rank has none
    (3, 400, 1024, 2.0, BF, False, True, ()),
    (3, 400, 1032, 4.0, F32, False, False, ()),
    (3, 400, 1032, 2.0, BF, False, True, (2, 3, 6)),
    (3, 130, 1032, 2.0, BF, False, True, ())])
def test_clusters_share_a_channel_tile(case):
    """Carry and adjoint from rank to rank: final state and dh0 to the 1e-5 of two-term operands, outputs in 16 bits as close as
    elsewhere in the tensor-core form.  The form word names the walk."""
    B, T, D, fs, gdt, utm, states, deep = case
    (y, hT, g, forms), (yo, hTo, go) = _run(B, T, D, fs, gdt, utm, states, f_logit=_deep(deep, slice(100, 140)) if deep else None)
    few = B * ((D + 127) // 128) * 4 < 148
    assert forms == {"fwd": WALK, "bwd": RECURRENT if deep or few else WALK}
    assert _err(hT, hTo) < 2e-5
    assert _err(y, yo) < 1e-3
    for k in g:
        assert _err(g[k], go[k]) < (2e-5 if k == "dh0" else 2e-3), k


@pytest.mark.parametrize("case", [(2, 64, 256, TICKET), (2, 1000, 384, TICKET), (1, 4096, 2048, WALK), (8, 128, 2048, WALK), (1, 130, 4736, WALK)])
def test_the_form_word_names_the_kernel_that_ran(case):
    """The ticket kernel where few channel tiles make a chain of chunks, a walk (by single CTAs, or by clusters) everywhere else."""
    from naju_b200 import naju_scan
    from naju_b200.scan import last_kernel_forms
    B, T, D, form = case
    r = lambda *s: torch.randn(*s, device="cuda", dtype=F32).to(BF)  # noqa: E731
    with torch.no_grad():
        naju_scan(r(B, T, D), r(B, T, D) + 2, r(B, T, D), r(B, T, 16), r(B, T, 16), torch.zeros(D, device="cuda"))
    assert last_kernel_forms()["fwd"] == form
