"""Selective scan on either side of each line between its kernels: tiles with too few live lanes, rows that the lanes fetch in one pass
or cut into segments, groups of a few channels, four warps per channel or one."""
import ctypes

import pytest
import torch

from helpers import TOL_BF16, TOL_FP32
from test_gpu_scan import make_inputs, run_both

DTYPES = [(torch.float32, TOL_FP32), (torch.bfloat16, TOL_BF16)]


@pytest.mark.parametrize("dim,groups,segments", [(2048, 1, 16), (2048, 64, 16), (2048, 256, 0), (2048, 128, 8), (1008, 42, 16), (1008, 63, 16), (1008, 126, 8)])
def test_segments_follow_the_tiles(dim, groups, segments):
    """A sequence is cut into as many segments as fill the GPU with tiles of 32 channels of ONE group (no GPU needed)."""
    from mamba_b200 import _build, _lib
    _build.build()
    a = _lib.ScanArgs()
    a.batch, a.dim, a.seqlen, a.dstate, a.ngroups, a.B_variable, a.C_variable = 1, dim, 2048, 16, groups, 1, 1
    need = ctypes.c_size_t(0)
    assert _lib.lib().mb200_scan_scratch_bytes(ctypes.byref(a), ctypes.byref(need)) == _lib.OK
    assert need.value == 3 * 4 * segments * dim * 16


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("batch,dim,L,N,groups", [
    (1, 1072, 139, 16, 1), (1, 1056, 139, 16, 1), (1, 4624, 501, 16, 1), (1, 4592, 501, 16, 1),     # one pass: steps against channels
    (2, 992, 101, 8, 1), (2, 984, 101, 8, 1), (1, 1600, 72, 8, 20), (1, 1680, 73, 8, 21),           # the same with few states
    (1, 2048, 72, 16, 256), (1, 1920, 72, 16, 128), (1, 2048, 73, 16, 128), (1, 2176, 72, 16, 128), # 8, 15, 16, 17 channels a group
    (2, 64, 72, 16, 64), (1, 1280, 33, 5, 1280),                                                    # one channel a group
    (1, 1040, 2051, 16, 1), (1, 2720, 1027, 16, 1), (1, 2640, 1027, 16, 1),                         # 16 segments; 8, either side
    (1, 14448, 40, 16, 602), (1, 14448, 41, 16, 602), (1, 21672, 40, 16, 903),                      # many CTAs, aligned and not
    (1, 592, 520, 16, 1), (1, 593, 520, 16, 1), (1, 296, 65, 16, 148), (1, 298, 65, 16, 149),       # four warps per channel, or one
])
def test_either_side(dtype, tol, batch, dim, L, N, groups):
    run_both(make_inputs(dim + L, batch, dim, L, N, groups, dtype, has_z=L != 73), tol, f"route b{batch} d{dim} L{L} N{N} G{groups}")
