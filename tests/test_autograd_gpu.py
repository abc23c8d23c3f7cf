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


def test_the_backward_keeps_the_forward_s_form(monkeypatch):
    """Fewer than 16 states are padded or not by NAJU_B200_FORM; the checkpoints of one layout are not read as the other's."""
    from naju_b200.scan import _desc, _prepare, scan_backward, scan_forward
    t = [x.requires_grad_(True) for x in _inputs(2, 512, 2048, 8, BF)]
    dy = torch.ones_like(t[0])
    want = torch.autograd.grad(_scan(t), t, dy)
    for first, then in (("auto", "recurrent"), ("recurrent", "auto")):
        monkeypatch.setenv("NAJU_B200_FORM", first)
        y = _scan(t)
        monkeypatch.setenv("NAJU_B200_FORM", then)
        for a, b in zip(torch.autograd.grad(y, t, dy), want):   # (two kernels apart: 16-bit operands, 2e-3 of bf16 gradients)
            assert ((a.double() - b.double()).norm() / b.double().norm()).item() < 2e-3
        # the raw calls name the mistake
        monkeypatch.setenv("NAJU_B200_FORM", first)
        p = _prepare(*[x.detach() for x in t[:6]])
        ckpt = scan_forward(*p)[3]
        monkeypatch.setenv("NAJU_B200_FORM", then)
        with pytest.raises(RuntimeError, match="NAJU_B200_FORM has changed"):
            scan_backward(_desc(*p[:5]), *p, None, dy, None, ckpt)


@pytest.mark.parametrize("which", range(7))
@pytest.mark.parametrize("grad", [True, False])
def test_forward_mode_is_refused(which, grad):
    """A dual input raises, as any autograd function without a jvp does; its tangent is not dropped."""
    import torch.autograd.forward_ad as fwAD
    t = _inputs()
    with fwAD.dual_level(), torch.set_grad_enabled(grad):
        t[which] = fwAD.make_dual(t[which], torch.ones_like(t[which]))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            _scan(t)


def test_function_transforms_are_refused():
    t = _inputs()
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda u: _scan([u] + t[1:]).sum())(t[0])
    with pytest.raises((RuntimeError, ValueError)):
        torch.func.vmap(lambda u: _scan([u] + t[1:]))(torch.stack([t[0], t[0]]))


@pytest.mark.parametrize("want_final", [False, True])
def test_compiled_autograd_around_an_eager_call(want_final):
    """The backward of an eager call under compiled autograd gives the eager backward's gradients."""
    t = [x.requires_grad_(True) for x in _inputs()]

    def loss():
        if not want_final:
            return _scan(t).square().mean()
        y, hT = _scan(t, return_final_state=True)
        return y.square().mean() + hT.square().mean()

    loss().backward()
    want = [x.grad.clone() for x in t]
    for x in t:
        x.grad = None
    with torch._dynamo.compiled_autograd._enable(torch.compile(backend="eager")):
        loss().backward()
    for x, w in zip(t, want):
        assert torch.allclose(x.grad, w, rtol=1e-5, atol=1e-8)


def test_saved_tensors_and_a_second_backward():
    """Saved-tensor hooks see what the node saves; a second backward without retain_graph is refused, with it repeats itself."""
    t = [x.requires_grad_(True) for x in _inputs()]
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda x: seen.append(x) or x.cpu(), lambda x: x.cuda()):
        y = _scan(t)
    assert len(seen) == 8
    a = torch.autograd.grad(y.sum(), t, retain_graph=True)
    b = torch.autograd.grad(y.sum(), t)
    for p, q in zip(a, b):
        assert torch.allclose(p, q, rtol=1e-5, atol=1e-7)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(y.sum(), t)


@pytest.mark.parametrize("state", [False, True])
def test_a_traced_scan_computes(state):
    """torch.jit.trace records the scan, not the allocation of its outputs: on other inputs the traced function gives the eager
    results, and their gradients."""
    import warnings
    from naju_b200 import naju_scan
    from naju_b200.scan import naju_b200_scan

    def fn(u, fl, il, B, C, D, h0):
        if state:
            y, hT = naju_scan(u * 2.0, fl, il, B, C, D, h0=h0, return_final_state=True)
            return y, hT
        return naju_scan(u * 2.0, fl, il, B, C, D) + naju_b200_scan(u, fl, il, B, C, D)

    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        traced = torch.jit.trace(fn, tuple(_inputs(seed=1)), check_trace=False)
    a, b = ([x.requires_grad_(True) for x in _inputs(seed=2)] for _ in range(2))
    out, want = traced(*a), fn(*b)
    out, want = (out, want) if state else ((out,), (want,))
    for x, y in zip(out, want):
        assert torch.allclose(x, y, rtol=1e-5, atol=1e-5)
    sum(x.square().mean() for x in out).backward()
    sum(x.square().mean() for x in want).backward()
    for x, y in zip(a[:6 + state], b):
        assert torch.allclose(x.grad, y.grad, rtol=1e-4, atol=1e-7)
