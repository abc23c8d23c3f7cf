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
