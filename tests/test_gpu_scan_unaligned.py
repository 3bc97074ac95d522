"""The channel-parallel scan over rows that TMA cannot describe: every shift of a row against 16-byte granules, ragged channel
groups, lengths around a hand-off (8 steps) and a tile, each layout of the kernel, a cut sequence, and the second (pre-gate) output."""
import pytest
import torch

import oracle
from helpers import TOL_BF16, TOL_FP32, assert_close
from test_gpu_scan import make_inputs, run_both

pytestmark = pytest.mark.gpu
DEV = "cuda"
DTYPES = [(torch.float32, TOL_FP32), (torch.bfloat16, TOL_BF16), (torch.float16, TOL_BF16)]


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("batch,dim,L,N,groups", [(1, 1024, 1, 16, 1), (1, 1024, 7, 16, 2), (1, 1040, 9, 8, 2), (2, 2064, 17, 16, 1), (1, 1100, 131, 5, 11)])
def test_short_rows_and_ragged_groups(dtype, tol, batch, dim, L, N, groups):
    run_both(make_inputs(L * 7 + N, batch, dim, L, N, groups, dtype), tol, f"unaligned b{batch} d{dim} L{L}")


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("dim,L", [(1024, 139), (19008, 45), (30016, 43)])      # the second and third: four- and three-warp CTAs in 16 bits, six in fp32
@pytest.mark.parametrize("has_z", [True, False])
def test_layouts_by_grid_size(dtype, tol, dim, L, has_z):
    run_both(make_inputs(dim + L, 1, dim, L, 16, 1, dtype, has_z=has_z), tol, f"unaligned d{dim} L{L}")


@pytest.mark.parametrize("dtype,tol", DTYPES[:2])
@pytest.mark.parametrize("L", [1031, 1037])
def test_cut_sequence(dtype, tol, L):
    run_both(make_inputs(L, 1, 1024 + 16, L, 16, 1, dtype), tol, f"unaligned, cut, L{L}")


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("off", range(8))
def test_every_shift_of_the_rows(dtype, tol, off):
    """Rows at every offset inside wider buffers; the elements around an output row stay as they were."""
    from mamba_b200 import ops

    L = 37
    inp = make_inputs(off, 1, 1024, L, 16, 1, dtype)
    c = {k: v.to(DEV) for k, v in inp.items()}

    def inside(t, step):
        o = off * step % 8
        buf = torch.full((1, 1024, L + 24), 7.0, dtype=dtype, device=DEV)
        buf[:, :, o:o + L] = t
        return buf, buf[:, :, o:o + L]

    u, delta, z = (inside(c[k], step)[1] for k, step in (("u", 1), ("delta", 3), ("z", 5)))
    buf, out = inside(torch.zeros_like(c["u"]), 7)
    ops._selective_scan(u, delta, c["A"], c["B"], c["C"], c["D"], z, c["delta_bias"], True, out=out)
    want = oracle.selective_scan(inp["u"].float(), inp["delta"].float(), inp["A"], inp["B"].float(), inp["C"].float(), inp["D"], inp["z"].float(),
                                 inp["delta_bias"], delta_softplus=True)
    assert_close(out, want, tol, f"offset {off}")
    out.fill_(7.0)
    assert bool((buf == 7.0).all())


@pytest.mark.parametrize("dtype,tol", DTYPES)
def test_second_output(dtype, tol):
    from mamba_b200.compat import selective_scan_cuda
    inp = make_inputs(5, 1, 1024, 53, 16, 1, dtype)
    c = {k: v.to(DEV) for k, v in inp.items()}
    out, _, out_z = selective_scan_cuda.fwd(c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], True)
    for got, z in ((out, None), (out_z, inp["z"].float())):
        want = oracle.selective_scan(inp["u"].float(), inp["delta"].float(), inp["A"], inp["B"].float(), inp["C"].float(), inp["D"], z,
                                     inp["delta_bias"], delta_softplus=True)
        assert_close(got, want, tol, "gated" if z is not None else "ungated")


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("off", range(8))
@pytest.mark.parametrize("L,W", [(1, 2), (5, 4), (16, 3), (259, 4), (267, 2)])
def test_conv_rows(dtype, tol, off, L, W):
    """The convolution before the scan over rows at every offset, its carried states included."""
    from mamba_b200 import causal_conv1d_fn
    g = torch.Generator().manual_seed(off * 31 + L)
    x = torch.randn(2, 12, L, generator=g).to(dtype)
    w, b, init = torch.randn(12, W, generator=g), torch.randn(12, generator=g), torch.randn(2, 12, W - 1, generator=g).to(dtype)
    buf = torch.zeros(2, 12, L + 16, dtype=dtype, device=DEV)
    xd = buf[:, :, off:off + L]
    xd.copy_(x)
    for kw in ({}, {"initial_states": init}):
        want, fin = oracle.causal_conv1d(x.float(), w, b, activation="silu", return_final_states=True, **{k: v.float() for k, v in kw.items()})
        got, gfin = causal_conv1d_fn(xd, w.to(DEV), b.to(DEV), activation="silu", return_final_states=True, **{k: v.to(DEV) for k, v in kw.items()})
        assert_close(got, want, tol, f"conv offset {off} L {L}")
        assert_close(gfin, fin, tol, "final states")


@pytest.mark.parametrize("dtype,tol", DTYPES)
@pytest.mark.parametrize("batch,dim,L,N,groups", [(1, 1, 1, 1, 1), (2, 6, 511, 5, 2), (1, 296, 33, 16, 1), (1, 297, 513, 16, 1), (3, 198, 130, 8, 2)])
def test_few_channels(dtype, tol, batch, dim, L, N, groups):
    run_both(make_inputs(dim + L, batch, dim, L, N, groups, dtype, has_z=L != 33), tol, f"few channels b{batch} d{dim} L{L}")
