"""The chunked scan in fp32 where its tiles end: chunk, head and state sizes off 64, off 32 and off 4 (element
loads), packed sequences, and 16-bit calls of the same shapes."""
import pytest
import torch

from helpers import TOL_BF16, TOL_FP32, assert_close
from test_gpu_ssd import make, run_both
from test_gpu_ssd_tc_shapes import _c, _fn, _packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, TOL_FP32), (torch.bfloat16, TOL_BF16)])
@pytest.mark.parametrize("L,H,P,G,N,Q", [(1, 1, 4, 1, 4, 16), (97, 2, 36, 1, 20, 33), (130, 2, 65, 2, 33, 64), (257, 4, 68, 1, 132, 96), (70, 2, 7, 1, 5, 30)])
def test_tile_edges(dtype, tol, L, H, P, G, N, Q):
    run_both(make(700 + L, 2, L, H, P, G, N, dtype, has_z=L % 2 == 1, init=True), Q, tol, f"L{L} P{P} N{N} Q{Q}")


@pytest.mark.parametrize("P,N,Q", [(64, 64, 64), (36, 20, 33)])
def test_packed(P, N, Q):
    """Each sequence of a packed row equals the same sequence on its own."""
    inp, seq_idx, cu = _packed(720 + P, [3, 100, 33, 1, 64], 2, P, 1, N, torch.float32)
    c = {k: _c(v) for k, v in inp.items()}
    kw = dict(D=c["D"], dt_bias=c["dt_bias"], dt_softplus=True, return_final_states=True)
    out, fin, var = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], Q, z=c["z"], seq_idx=seq_idx.cuda(), cu_seqlens=cu.cuda(), return_varlen_states=True, **kw)
    for i in range(5):
        s = slice(int(cu[i]), int(cu[i + 1]))
        o, f = _fn()(c["x"][:, s], c["dt"][:, s], c["A"], c["B"][:, s], c["C"][:, s], Q, z=c["z"][:, s], **kw)
        assert_close(out[:, s], o, TOL_FP32, f"sequence {i}")
        assert_close(var[i:i + 1], f, TOL_FP32, f"end state {i}")
