"""The recurrent backward of 16 states, 16-bit inputs and logits and 64-step chunks against the fp64 oracle, at the edges of its tiles
(64 steps, 128 channels, eight steps between two partial sums)."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

RECURRENT = 1
BF, F16, F32 = torch.bfloat16, torch.float16, torch.float32


def _round(x, dt):
    return torch.tensor(x).to(dt).float().numpy()


# B, T, D, f_shift, type of u and the logits
@pytest.mark.parametrize("case", [
    (2, 1, 8, 2.0, BF), (2, 7, 136, 2.0, F16), (1, 63, 128, 2.0, BF), (2, 64, 264, 4.0, BF), (3, 65, 120, 2.0, F16), (2, 193, 1032, 2.0, BF),
    (1, 1000, 256, 4.0, BF),            # look-back over many chunks
    (2, 130, 256, -4.0, BF),            # deep gates: d f_logit from states walked again
    (3, 128, 20000, 2.0, BF)])          # more tiles than the GPU holds at once
def test_recurrent_backward_of_16_bit_tiles(case, monkeypatch):
    """Outputs in 16 bits differ from the identically rounded oracle by single roundings at most (1e-3); the fp32 ones (dD, dh0) are
    sums of fp32 products: 2e-6."""
    from naju_b200 import naju_scan
    from naju_b200.scan import last_kernel_forms
    monkeypatch.setenv("NAJU_B200_CHECK_STATUS", "1")
    monkeypatch.setenv("NAJU_B200_FORM", "recurrent")
    B, T, D, fs, dt = case
    d = oracle.make_inputs(B, T, D, 16, seed=9, f_shift=fs, d_skip_scale=0.05, with_h0=True)
    cast = {"u": dt, "fl": dt, "il": dt, "dy": dt, "Bm": BF, "Cm": BF}
    q = {k: (_round(d[k], cast[k]) if k in cast else d[k]) for k in d}
    t = {k: torch.tensor(q[k], device="cuda").to(cast.get(k, F32)) for k in q}
    x = {k: t[k].requires_grad_(True) for k in ("u", "fl", "il", "Bm", "Cm", "Dskip", "h0")}
    y, hT = naju_scan(*(x[k] for k in ("u", "fl", "il", "Bm", "Cm", "Dskip")), h0=x["h0"], return_final_state=True)
    torch.autograd.backward([y, hT], [t["dy"], t["dhT"]])
    torch.cuda.synchronize()
    assert last_kernel_forms() == {"fwd": RECURRENT, "bwd": RECURRENT}
    go = oracle.oracle_bwd(*(q[k] for k in ("u", "fl", "il", "Bm", "Cm", "Dskip")), q["dy"], h0=q["h0"], dhT=q["dhT"])
    for k, src in (("du", "u"), ("dfl", "fl"), ("dil", "il"), ("dB", "Bm"), ("dC", "Cm")):
        assert oracle.rel_l2(x[src].grad.float().cpu().numpy(), _round(go[k], cast[src])) < 1e-3, k
    assert oracle.rel_l2(x["Dskip"].grad.cpu().numpy(), go["dD"]) < 2e-6
    assert oracle.rel_l2(x["h0"].grad.cpu().numpy(), go["dh0"]) < 2e-6
