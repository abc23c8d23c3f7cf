"""The tensor-core kernels of 17 to 64 states against the fp64 oracle, at the edges of their tiles (32 steps, 128
channels, 16-step and 8-step slabs, state widths of 32 and 64)."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

WALK, RECURRENT = 3, 1
BF, F32 = torch.bfloat16, torch.float32


@pytest.fixture(autouse=True)
def _status_checks(monkeypatch):
    monkeypatch.setenv("NAJU_B200_CHECK_STATUS", "1")


def _round(x, dt):
    return torch.tensor(x).to(dt).float().numpy()


# B, T, D, N, f_shift, logits, time-contiguous u, fwd form, bwd form
@pytest.mark.parametrize("case", [
    (8, 1, 2432, 64, 2.0, BF, False, WALK, WALK),          # one step
    (8, 31, 2432, 64, 2.0, BF, False, WALK, WALK),         # one short chunk
    (4, 73, 4360, 64, 2.0, BF, False, WALK, WALK),         # ragged end, partial channel tile (D % 128 = 8)
    (5, 96, 4096, 40, 4.0, BF, False, WALK, WALK),         # more channel tiles than SMs, padded states
    (6, 104, 2560, 24, 2.0, BF, True, WALK, WALK),         # time-contiguous u, 32-state kernels
    (6, 67, 2560, 32, 2.0, F32, False, WALK, RECURRENT),   # fp32 logits keep the recurrent backward
    (6, 96, 2560, 64, 0.0, BF, False, WALK, WALK),         # retention about one half
    (6, 96, 2560, 64, -3.0, BF, False, WALK, RECURRENT),   # deep gates: exact tiles, recurrent backward
    (6, 96, 2560, 20, 2.0, BF, False, RECURRENT, RECURRENT),   # rows of B / C that TMA cannot describe
    (1, 2048, 256, 64, 2.0, BF, False, RECURRENT, RECURRENT)])  # too few channel tiles
def test_wide_state_kernels_match_the_oracle(case):
    """16-bit outputs against the identically rounded oracle; the fp32 ones (final state, dD, dh0, and dfl with fp32
    logits) to 1e-6, which the recurrent kernels' 1e-7 to 2e-7 leaves room for and a two-term operand (1e-5) would not."""
    from naju_b200 import naju_scan
    from naju_b200.scan import last_kernel_forms
    B, T, D, N, fs, gdt, utm, ffwd, fbwd = case
    d = oracle.make_inputs(B, T, D, N, seed=5, f_shift=fs, d_skip_scale=0.05, with_h0=True)
    cast = {"u": BF, "Bm": BF, "Cm": BF, "dy": BF, "fl": gdt, "il": gdt}
    q = {k: (_round(d[k], cast[k]) if k in cast else d[k]) for k in d}
    t = {k: torch.tensor(q[k], device="cuda").to(cast.get(k, F32)) for k in ("u", "fl", "il", "Bm", "Cm", "Dskip", "h0")}
    if utm:
        t["u"] = t["u"].transpose(1, 2).contiguous().transpose(1, 2)
    for k in t:
        t[k].requires_grad_(True)
    y, hT = naju_scan(t["u"], t["fl"], t["il"], t["Bm"], t["Cm"], t["Dskip"], h0=t["h0"], return_final_state=True)
    torch.autograd.backward([y, hT], [torch.tensor(q["dy"], device="cuda").to(BF), torch.tensor(d["dhT"], device="cuda")])
    torch.cuda.synchronize()
    assert last_kernel_forms() == {"fwd": ffwd, "bwd": fbwd}
    a = (q["u"], q["fl"], q["il"], q["Bm"], q["Cm"], q["Dskip"])
    yo, hTo = oracle.oracle_fwd(*a, h0=q["h0"], return_final_state=True)
    g = oracle.oracle_bwd(*a, q["dy"], h0=q["h0"], dhT=d["dhT"])
    assert oracle.rel_l2(y.detach().float().cpu().numpy(), _round(yo, BF)) < 1e-3
    assert oracle.rel_l2(hT.detach().cpu().numpy(), hTo) < 1e-6
    for k, src in (("du", "u"), ("dfl", "fl"), ("dil", "il"), ("dB", "Bm"), ("dC", "Cm")):
        ref = _round(g[k], gdt if k in ("dfl", "dil") else BF)
        assert oracle.rel_l2(t[src].grad.float().cpu().numpy(), ref) < 2e-3, k
    assert oracle.rel_l2(t["Dskip"].grad.cpu().numpy(), g["dD"]) < 1e-6
    assert oracle.rel_l2(t["h0"].grad.cpu().numpy(), g["dh0"]) < 1e-6


def _inputs(B, T, D, N, f_shift, utm=False, seed=11, **kw):
    d = oracle.make_inputs(B, T, D, N, seed=seed, f_shift=f_shift, **kw)
    cast = {"u": BF, "Bm": BF, "Cm": BF, "dy": BF, "fl": BF, "il": BF}
    q = {k: (_round(d[k], cast[k]) if k in cast else d[k]) for k in d}
    t = {k: torch.tensor(q[k], device="cuda").to(cast.get(k, F32)) for k in q}
    if utm:
        t["u"] = t["u"].transpose(1, 2).contiguous().transpose(1, 2)
    return q, t


ORDER = ("u", "fl", "il", "Bm", "Cm", "Dskip")


def _run(t, dhT=True):
    """y, hT and the gradients of ORDER and h0, with the kernel forms that made them."""
    from naju_b200 import naju_scan
    from naju_b200.scan import last_kernel_forms
    x = {k: t[k].detach().requires_grad_(True) for k in ORDER + ("h0",)}
    y, hT = naju_scan(*(x[k] for k in ORDER), h0=x["h0"], return_final_state=True)
    torch.autograd.backward([y, hT], [t["dy"], t["dhT"] if dhT else torch.zeros_like(hT)])
    torch.cuda.synchronize()
    return y.detach(), hT.detach(), {k: x[k].grad for k in x}, last_kernel_forms()


# B, T, D, N, f_shift, time-contiguous u
@pytest.mark.parametrize("case", [(6, 200, 2560, 64, 2.0, False), (6, 200, 2560, 64, 5.0, True), (7, 199, 2568, 32, 2.0, False)])
def test_wide_state_kernels_compute_in_fp32(case, monkeypatch):
    """What is rounded to 16 bits at the end is fp32 until then.  Three bf16 terms hold 24 bits, and some 60 accumulating MMAs that
    truncate leave about 1e-6; where two values 1e-6 apart are rounded to bf16 (steps of 2^-8) one pair in 2000 lands a step apart,
    6e-5 in the 2-norm.  (Operands of two terms, 16 bits: 4e-4.)  The fp32 results are no further off than the recurrent
    kernels' (up to what a different order of the sums makes of 2560 x 64 roundings, 2 %)."""
    B, T, D, N, fs, utm = case
    q, t = _inputs(B, T, D, N, fs, utm, d_skip_scale=0.05, with_h0=True)
    y, hT, g, forms = _run(t)
    assert forms == {"fwd": WALK, "bwd": WALK}
    a = tuple(q[k] for k in ORDER)
    yo, hTo = oracle.oracle_fwd(*a, h0=q["h0"], return_final_state=True)
    go = oracle.oracle_bwd(*a, q["dy"], h0=q["h0"], dhT=q["dhT"])
    assert oracle.rel_l2(y.float().cpu().numpy(), _round(yo, BF)) < 1e-4
    for k, src in (("du", "u"), ("dfl", "fl"), ("dil", "il"), ("dB", "Bm"), ("dC", "Cm")):
        assert oracle.rel_l2(g[src].float().cpu().numpy(), _round(go[k], BF)) < 1e-4, k
    monkeypatch.setenv("NAJU_B200_FORM", "recurrent")
    _, hT_r, g_r, forms = _run(t)
    assert forms == {"fwd": RECURRENT, "bwd": RECURRENT}
    for name, ours, theirs, want in (("hT", hT, hT_r, hTo), ("dh0", g["h0"], g_r["h0"], go["dh0"])):
        err, err_r = (oracle.rel_l2(v.cpu().numpy(), want) for v in (ours, theirs))
        assert err <= 1.02 * err_r, (name, err, err_r)


@pytest.mark.parametrize("utm", [False, True])
def test_wide_state_write_gates_near_zero(utm):
    """sigmoid(-40) is 4e-18 and sigmoid(-70) 4e-31, also next to gates of ordinary size and in the gradients.  (1e-3: as above, but
    the outputs of a third of the channels at a time.)"""
    B, T, D, N = 6, 96, 2560, 64
    q, t = _inputs(B, T, D, N, 2.0, utm, with_h0=True)
    low = torch.zeros(D, device="cuda")
    low[::3], low[1::3] = -40.0, -70.0
    t["il"] = (t["il"].float() + low).to(BF)
    t["h0"], t["dhT"] = torch.zeros_like(t["h0"]), torch.zeros_like(t["dhT"])
    q["il"], q["h0"], q["dhT"] = t["il"].float().cpu().numpy(), t["h0"].cpu().numpy(), t["dhT"].cpu().numpy()
    y, _, g, forms = _run(t, dhT=False)
    assert forms == {"fwd": WALK, "bwd": WALK}
    a = tuple(q[k] for k in ORDER)
    yo = oracle.oracle_fwd(*a, h0=q["h0"])
    go = oracle.oracle_bwd(*a, q["dy"], h0=q["h0"], dhT=q["dhT"])
    for name, ours, want in (("y", y, yo), ("du", g["u"], go["du"]), ("dfl", g["fl"], go["dfl"]), ("dil", g["il"], go["dil"])):
        for k in range(3):
            assert oracle.rel_l2(ours[..., k::3].double().cpu().numpy() * 1e15, _round(want[..., k::3], BF).astype("f8") * 1e15) < 1e-3, (name, k)


@pytest.mark.parametrize("where", ["u", "Bm", "Cm", "h0", "fl", "dy", "dhT", "huge u", "huge B", "huge dy"])
def test_wide_state_kernels_keep_what_is_not_finite_where_it_belongs(where, monkeypatch):
    """An infinity or NaN reaches the steps after it (or, in the backward, before it) and the state, channel and batch row it
    belongs to, exactly as in the recurrent kernels; everything else is as finite as there and the same up to a rounding."""
    B, T, D, N = 6, 104, 2560, 64
    _, t = _inputs(B, T, D, N, 2.0, with_h0=True)
    inf = float("inf")
    if where in ("u", "dy"):
        t[where][1, 41, 7], t[where][2, 70, 300] = inf, float("nan")
    elif where == "huge u":
        t["u"][1, 41, 7] = 1e37
    elif where == "huge B":
        t["Bm"][1, 41, 7], t["Cm"][2, 41, 7] = 1e30, -1e30
    elif where == "huge dy":
        t["dy"][1, 41, 7] = -1e30
    elif where in ("Bm", "Cm"):
        t[where][1, 41, 7] = -inf
    elif where == "fl":
        t[where][1, 41, 7], t[where][2, 41, 9] = float("nan"), -inf
    else:
        t[where][1, 300, 7] = inf
    y, hT, g, forms = _run(t)
    assert forms["bwd"] == RECURRENT   # (by the forward's mark, or because the tensor-core backward hands the work on)
    monkeypatch.setenv("NAJU_B200_FORM", "recurrent")
    y_r, hT_r, g_r, _ = _run(t)
    for name, a, b in [("y", y, y_r), ("hT", hT, hT_r)] + [(k, g[k], g_r[k]) for k in g]:
        assert torch.equal(torch.isnan(a), torch.isnan(b)), name
        assert torch.equal(torch.isinf(a), torch.isinf(b)), name
        both = torch.isfinite(a) & torch.isfinite(b)
        assert bool(both.any()) and oracle.rel_l2(a[both].double().cpu().numpy(), b[both].double().cpu().numpy()) < 4e-3, name


def test_wide_state_d_skip_gradient_over_a_long_sequence():
    """dD = sum dy u over 8192 steps of equal products: one running sum of every fourth octet loses 2e-5 to one-sided roundings; sums
    per chunk, added up with what the additions drop, stay at fp32's own 6e-8 a value."""
    from naju_b200 import naju_scan
    from naju_b200.scan import last_kernel_forms
    B, T, D, N = 1, 8192, 6400, 24
    gen = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    u, dy = ((torch.rand(D, device="cuda", generator=gen) + 0.5).to(BF).expand(B, T, D).contiguous() for _ in range(2))
    skip = r(D).requires_grad_(True)
    y = naju_scan(u, (r(B, T, D) + 2).to(BF), r(B, T, D).to(BF), r(B, T, N).to(BF), r(B, T, N).to(BF), skip)
    dD, = torch.autograd.grad(y, [skip], [dy])
    assert last_kernel_forms()["bwd"] == WALK
    want = (dy.double() * u.double()).sum((0, 1))
    assert ((dD.double() - want).norm() / want.norm()).item() < 2e-7
