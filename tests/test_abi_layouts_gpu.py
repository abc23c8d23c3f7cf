"""Layouts that the C ABI takes and the Python layer never hands on: a time-contiguous u (and du) whose channel stride, batch stride
or base is no multiple of 16 bytes."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

BF, F32 = torch.bfloat16, torch.float32


def _p(t):
    return None if t is None else t.data_ptr()


# u_sd beyond T, elements before the first of u and of du
@pytest.mark.parametrize("pad,u_off,du_off", [(0, 0, 0), (1, 0, 0), (2, 1, 3), (3, 2, 0), (4, 0, 1), (7, 5, 0)])
@pytest.mark.parametrize("T", [45, 64])
@pytest.mark.parametrize("dtypes", [(F32, F32), (BF, F32), (BF, BF)])
def test_time_contiguous_u_of_any_alignment(dtypes, T, pad, u_off, du_off):
    """Against the same call on a channel-contiguous copy: the same kernels up to the order of fp32 sums (2e-6), rounded to 16 bits a
    step apart in one place of 2000 (7e-5)."""
    from naju_b200 import _lib
    lib = _lib.load()
    act, gate = dtypes
    B, D, N = 2, 136, 16
    gen = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    u_sd = T + pad
    u_sb = D * u_sd + pad
    u, fl, il, dy = r(B, T, D).to(act), (r(B, T, D) + 2).to(gate), r(B, T, D).to(gate), r(B, T, D).to(act)
    Bm, Cm, skip = r(B, T, N).to(act), r(B, T, N).to(act), r(D)
    stream = torch.cuda.current_stream().cuda_stream
    size = B * u_sb + 64
    strided = lambda buf, off: buf.as_strided((B, T, D), (u_sb, 1, u_sd), off)  # noqa: E731
    u_buf, du_buf = (torch.full((size,), float("nan"), device="cuda", dtype=act) for _ in range(2))
    strided(u_buf, u_off).copy_(u)

    def call(time_contiguous):
        d = _lib.ScanDesc()
        d.B, d.T, d.D, d.N = B, T, D, N
        code = {F32: _lib.NAJU_F32, BF: _lib.NAJU_BF16}
        d.act_dtype, d.gate_dtype, d.bc_dtype = code[act], code[gate], code[act]
        d.flags = _lib.FLAG_RECURRENT_ONLY
        d.fl_sb = d.il_sb = d.u_sb = T * D
        d.fl_st = d.il_st = d.u_st = D
        d.bm_sb = d.cm_sb = T * N
        d.bm_st = d.cm_st = N
        pu = u.data_ptr()
        if time_contiguous:
            d.u_sb, d.u_st, d.u_sd = u_sb, 1, u_sd
            pu = u_buf[u_off:].data_ptr()
        new = lambda t: torch.full_like(t, float("nan"))  # noqa: E731
        work = lambda n: torch.empty(int(n), dtype=torch.uint8, device="cuda")  # noqa: E731
        y, hT, ck, sc = new(u), r(B, D, N), work(lib.naju_b200_ckpt_bytes(d)), work(lib.naju_b200_fwd_scratch_bytes(d))
        args = [_p(fl), _p(il), _p(Bm), _p(Cm), _p(skip), None]
        rc = lib.naju_b200_fwd(d, pu, *args, _p(y), _p(hT), None, _p(ck), _p(sc), stream)
        assert rc == 0, _lib.strerror(rc)
        g = {"du": new(u), "dfl": new(fl), "dil": new(il), "dB": new(Bm), "dC": new(Cm), "dD": new(skip)}
        out = [_p(v) for v in g.values()]
        if time_contiguous:
            out[0] = du_buf[du_off:].data_ptr()
        sc = work(lib.naju_b200_bwd_scratch_bytes(d))
        rc = lib.naju_b200_bwd(d, pu, *args, _p(dy), None, _p(ck), *out, None, _p(sc), stream)
        assert rc == 0, _lib.strerror(rc)
        torch.cuda.synchronize()
        assert lib.naju_b200_read_status(_p(sc), stream) == 0
        if time_contiguous:
            g["du"] = strided(du_buf, du_off).contiguous()
        return {"y": y, "hT": hT, **g}

    want, got = call(False), call(True)
    for k in want:
        tol = 2e-6 if want[k].dtype == F32 else 7e-5
        assert oracle.rel_l2(got[k].float().cpu().numpy(), want[k].float().cpu().numpy()) < tol, k
    # nothing outside du's own elements was written
    mask = torch.ones(size, dtype=torch.bool, device="cuda")
    strided(mask, du_off).fill_(False)
    assert bool(torch.isnan(du_buf[mask]).all())


@pytest.mark.parametrize("case", [(2, 6000, 1000, 16, F32, F32), (3, 4100, 1001, 16, BF, BF), (1, 9000, 700, 24, F32, F32), (1, 9100, 700, 24, BF, F32)])
def test_noalloc_forward_of_problems_that_need_long_chunks(case):
    """Above half of the built-in array the recurrent kernels take chunks of 64 steps: the results of the caller-workspace call with
    its 32, up to the order of fp32 sums."""
    from naju_b200 import _lib
    from naju_b200.scan import _desc, scan_forward
    lib = _lib.load()
    B, T, D, N, act, gate = case
    gen = torch.Generator(device="cuda").manual_seed(8)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    t = [r(B, T, D).to(act), (r(B, T, D) + 4).to(gate), r(B, T, D).to(gate), (r(B, T, N) / 4).to(act), (r(B, T, N) / 4).to(act), r(D)]
    h0 = r(B, D, N)
    d = _desc(*t[:5])
    assert lib.naju_b200_ckpt_bytes(d) + lib.naju_b200_fwd_scratch_bytes(d) > _lib.NOALLOC_BYTES
    stream = torch.cuda.current_stream().cuda_stream
    y, hT = torch.full_like(t[0], float("nan")), torch.full_like(h0, float("nan"))
    rc = lib.naju_b200_fwd_noalloc(d, *map(_p, t), _p(h0), _p(y), _p(hT), stream)
    assert rc == 0, _lib.strerror(rc)
    torch.cuda.synchronize()
    assert lib.naju_b200_noalloc_read_status(stream) == 0 and lib.naju_b200_noalloc_read_form(stream) == _lib.FORM_RECURRENT
    y_ref, hT_ref, *_ = scan_forward(*t, h0, want_final=True)
    assert oracle.rel_l2(hT.cpu().numpy(), hT_ref.cpu().numpy()) < 2e-6
    assert oracle.rel_l2(y.float().cpu().numpy(), y_ref.float().cpu().numpy()) < (2e-6 if act == F32 else 7e-5)
