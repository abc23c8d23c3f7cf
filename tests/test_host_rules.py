"""Rules that the host layer states twice, in C++ and in Python (CPU only)."""
import itertools

import pytest
import torch

BF, F16, F32 = torch.bfloat16, torch.float16, torch.float32


@pytest.fixture(scope="module")
def lib():
    from naju_b200.build import build
    build()
    from naju_b200 import _lib
    return _lib.load()


def test_fake_checkpoint_size_is_the_library_s(lib):
    """torch.compile asserts the sizes that a custom op's fake implementation promises: the checkpoint buffer's is the library's for
    every type, state width and number of channels, padding of fewer than 16 states included."""
    from naju_b200 import _lib
    from naju_b200.scan import _ckpt_bytes_formula, _pads_to_group
    code = {F32: _lib.NAJU_F32, BF: _lib.NAJU_BF16, F16: _lib.NAJU_F16}
    for (B, T), D, N, act, bdt in itertools.product([(1, 1), (2, 300), (4, 520), (3, 1021)], [1, 100, 1000, 1001, 2050, 2434, 2440],
                                                    [1, 8, 15, 16, 17, 24, 32, 64, 128], [F32, BF, F16], [F32, BF, F16]):
        d = _lib.ScanDesc()
        d.B, d.T, d.D = B, T, D
        d.N = 16 if _pads_to_group(B * T * D, T, N, act, bdt) else N
        d.act_dtype = d.gate_dtype = code[act]
        d.bc_dtype = code[bdt]
        assert _ckpt_bytes_formula(B, T, D, d.N, act, bdt) == lib.naju_b200_ckpt_bytes(d), (B, T, D, N, act, bdt)


@pytest.mark.parametrize("D,N,act,bdt", [(1024, 16, F32, F32), (1000, 8, F32, F32), (1001, 16, BF, BF), (1024, 16, BF, BF), (512, 12, F16, F32),
                                         (768, 24, BF, BF), (768, 32, F32, F32), (768, 64, F32, F32)])
def test_noalloc_takes_problems_up_to_its_array(lib, D, N, act, bdt):
    """Chunk-boundary states and aggregates of 64-step chunks (32 above 32 states) are what has to fit in 32 MiB; nothing below that is
    refused as too large, everything above is.  (Refused before any CUDA call; what is accepted ends at the NULL pointers, or
    here, without a GPU, at the first CUDA call.)"""
    from naju_b200 import _lib
    code = {F32: _lib.NAJU_F32, BF: _lib.NAJU_BF16, F16: _lib.NAJU_F16}
    up = lambda x: (x + 255) // 256 * 256  # noqa: E731
    NS, step = (16, 64) if N <= 16 else (32, 64) if N <= 32 else (64, 32)

    def need(T):
        tiles = (T + step - 1) // step * 2 * ((D + 127) // 128)
        ckpt = up(tiles * 128 * NS * 4) + up(tiles * 128 * 4) + 256
        return ckpt + 256 + up(tiles * 4) + up(tiles * 128 * 4) + up(tiles * 128 * NS * 4)

    T = step
    while need(T + step) <= _lib.NOALLOC_BYTES:
        T += step
    for steps, refused in ((T, False), (T + 1, True)):
        d = _lib.ScanDesc()
        d.B, d.T, d.D, d.N = 2, steps, D, N
        d.act_dtype = d.gate_dtype = code[act]
        d.bc_dtype = code[bdt]
        d.u_sb = d.fl_sb = d.il_sb = steps * D
        d.u_st = d.fl_st = d.il_st = D
        d.bm_sb = d.cm_sb = steps * N
        d.bm_st = d.cm_st = N
        rc = lib.naju_b200_fwd_noalloc(d, *([None] * 10))
        assert (rc == _lib.E_TOO_LARGE) == refused, (steps, rc)
