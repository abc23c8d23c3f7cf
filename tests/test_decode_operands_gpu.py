"""Row operands of the decode step in the layouts a caller may have them in."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("which", ["u", "f_logit", "i_logit", "B", "C", "all"])
@pytest.mark.parametrize("layout", ["expanded", "overlapping", "columns", "wide rows"])
def test_decode_step_takes_its_operands_in_any_layout(layout, which, batch):
    """Broadcast over the batch (stride 0), rows that overlap, columns of another tensor, rows with a gap: the results of contiguous
    copies, bit for bit."""
    from naju_b200 import naju_scan_step
    D, N = 72, 16
    g = torch.Generator(device="cuda").manual_seed(6)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731

    def make(n):
        if layout == "expanded":
            return r(1, n).expand(batch, n)
        if layout == "overlapping":
            return r(n + 8 * batch).as_strided((batch, n), (8, 1))
        if layout == "columns":
            return r(n, batch).t()
        return r(batch, n + 5)[:, :n]

    names = {"u": D, "f_logit": D, "i_logit": D, "B": N, "C": N}
    ops = {k: make(n) if which in (k, "all") else r(batch, n) for k, n in names.items()}
    skip, state = r(D), r(batch, D, N)
    s1, s2 = state.clone(), state.clone()
    y1, _ = naju_scan_step(s1, *ops.values(), skip)
    y2, _ = naju_scan_step(s2, *(v.contiguous() for v in ops.values()), skip)
    assert torch.equal(y1, y2) and torch.equal(s1, s2)
