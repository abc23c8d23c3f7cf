"""What autograd, and the tools that look into it, get from the scan's native node."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF, F32 = torch.bfloat16, torch.float32


def _inputs(B=2, T=130, D=72, N=16, act=F32, seed=5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    return [r(B, T, D).to(act), (r(B, T, D) + 2).to(act), r(B, T, D).to(act), (r(B, T, N) / 4).to(act), (r(B, T, N) / 4).to(act), r(D),
            r(B, D, N)]


def _scan(t, **kw):
    from naju_b200 import naju_scan
    return naju_scan(*t[:6], h0=t[6] if len(t) > 6 else None, **kw)


@pytest.mark.parametrize("which", range(7))
def test_a_change_in_place_before_the_backward_is_noticed(which):
    """Every input that the backward reads, the initial state and D_skip (fp32, kept as they are) among them."""
    t = [x.requires_grad_(i != which) for i, x in enumerate(_inputs())]
    y = _scan(t)
    with torch.no_grad():
        t[which].add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
