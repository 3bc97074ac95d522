"""The SSD stages for 16-bit inputs at the edges of what they take: heads and states that do not fill a tile, lengths either side of a
row block and a chunk, other chunk sizes, few heads over many chunks, packed sequences on every one of them.  Headdim 64, dstate 128 and
chunk 256 run on 16-bit operands, all else on split ones (whose precision test_gpu_ssd_split.py checks)."""
import pytest
import torch

import oracle
from helpers import TOL_BF16, assert_close
from test_gpu_ssd import DEV, _c, _fn, _packed, _status, make, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("P,N,G,H,D_hdim", [(64, 64, 1, 6, False), (128, 128, 2, 4, True), (128, 64, 1, 3, False), (40, 24, 1, 5, True), (8, 8, 2, 2, False),
                                            (256, 96, 1, 2, True), (72, 128, 1, 2, False)])
def test_head_and_state_sizes(dtype, P, N, G, H, D_hdim):
    run_both(make(300 + P + N, 2, 300, H, P, G, N, dtype, D_hdim=D_hdim, init=True), 256, TOL_BF16, f"P{P} N{N}")


@pytest.mark.parametrize("L", [1, 127, 128, 129, 255, 256, 257, 384, 385, 640])
def test_lengths_around_row_blocks_and_chunks(L):
    run_both(make(320 + L, 1, L, 4, 64, 2, 128, torch.bfloat16, has_z=L % 2 == 0), 256, TOL_BF16, f"L{L}")


@pytest.mark.parametrize("has_z", [True, False])
@pytest.mark.parametrize("L,G", [(356, 1), (257, 1), (384, 1), (356, 80), (100, 80), (100, 1)])
def test_rows_after_a_short_last_chunk(L, G, has_z):
    """A last chunk of up to 128 steps has nothing for the warps of its lower row block, which reach the next batch row's first chunk while the
    heads of the short one are in flight.  Each of 148 CTAs has six or seven heads here, those that come to a new row three or five of the row before;
    with a group per head, every one has its own C and B, and with 100 steps there is nothing for those warps at all."""
    run_both(make(350 + L, 6, L, 80, 64, G, 128, torch.bfloat16, has_z=has_z), 256, TOL_BF16, f"L{L} G{G} z {has_z}")


@pytest.mark.parametrize("Q", [32, 64, 128, 512])
@pytest.mark.parametrize("N", [64, 128])
def test_other_chunk_sizes(Q, N):
    run_both(make(340 + Q, 2, 700, 4, 64, 1, N, torch.bfloat16, init=True), Q, TOL_BF16, f"Q{Q} N{N}")


@pytest.mark.parametrize("P,N,H", [(64, 128, 2), (128, 64, 1), (64, 96, 3)])
def test_few_heads_over_many_chunks(P, N, H):
    """Fewer than 74 head slices and more than eight chunks: chunk states side by side, recurrence in a launch of its own."""
    run_both(make(360 + N, 1, 2600, H, P, 1, N, torch.bfloat16, init=True), 256, TOL_BF16, f"few heads P{P} N{N}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("A", [-60.0, -400.0, -4000.0])
def test_decays_steeper_than_the_factorised_mask(dtype, A):
    inp = make(370, 1, 300, 3, 64, 1, 64, dtype)
    inp["A"] = torch.tensor([A, -2.0, 0.5 * A])
    run_both(inp, 256, TOL_BF16, f"A {A}")


@pytest.mark.parametrize("dtype,tie", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)])
def test_weight_of_a_step_on_itself(dtype, tie):
    """On 16-bit operands: dt, though it is formed with two exponents from sums of up to 500.  Here it lies 1e-6 below the middle between 1 and the
    next number of the input type and has to be rounded to 1; two exponentials of 2^-22 do not reach that middle, half an ulp of the sums does.
    Inputs 73 steps apart, at every place of eight, so that what came before has decayed to nothing."""
    L, H = 73 * 64, 2
    x, B = torch.zeros(1, L, H, 64, dtype=dtype), torch.zeros(1, L, 1, 128, dtype=dtype)
    x[:, ::73] = 1.0
    B[..., 0] = 1.0
    dt, A = torch.full((1, L, H), (1.0 + tie) * (1 - 1e-6)), torch.tensor([-0.7, -1.3])
    out = _fn()(*(_c(t) for t in (x, dt, A, B, B)), 256).cpu()
    assert _status() == 0 and torch.equal(out[:, ::73], x[:, ::73])


@pytest.mark.parametrize("P,N,H,lens", [(64, 64, 4, [100, 156, 1, 300, 40]), (128, 128, 2, [257, 255, 130]), (40, 24, 2, [3, 128, 200]),
                                        (64, 128, 2, [1000, 1, 1400, 128])])
def test_packed_sequences_and_their_end_states(P, N, H, lens):
    inp, seq_idx, cu = _packed(380 + N, lens, H, P, 1, N, torch.bfloat16)
    c = {k: _c(v) for k, v in inp.items()}
    out, fin, var = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 128, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], seq_idx=seq_idx.to(DEV),
                          cu_seqlens=cu.to(DEV), dt_softplus=True, return_final_states=True, return_varlen_states=True)
    assert _status() == 0
    f = lambda t: t.float()
    for i in range(len(lens)):
        sl = slice(int(cu[i]), int(cu[i + 1]))
        want, wfin = oracle.ssd_chunk_scan(f(inp["x"][:, sl]), f(inp["dt"][:, sl]), inp["A"], f(inp["B"][:, sl]), f(inp["C"][:, sl]), 128, inp["D"],
                                           f(inp["z"][:, sl]), inp["dt_bias"], None, dt_softplus=True)
        assert_close(out[:, sl], want, TOL_BF16, f"packed out seq {i}")
        assert_close(var[i:i + 1], wfin, TOL_BF16, f"varlen state seq {i}")
    assert_close(fin, var[-1:], TOL_BF16, "final state is the last sequence's")


@pytest.mark.parametrize("L", [296 * 256, 297 * 256 - 5])
def test_packed_row_on_both_sides_of_the_wide_prefix_sum(L):
    """More chunks than the 32-warp prefix-sum kernel is used for: each sequence of a packed row equals the same sequence on its own."""
    lens = [100, 40000, 1, L - 40101]
    inp, seq_idx, cu = _packed(400, lens, 2, 64, 1, 64, torch.bfloat16)
    c = {k: _c(v) for k, v in inp.items()}
    kw = dict(D=c["D"], dt_bias=c["dt_bias"], dt_softplus=True)
    out = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, z=c["z"], seq_idx=seq_idx.to(DEV), **kw)
    for i in range(len(lens)):
        s = slice(int(cu[i]), int(cu[i + 1]))
        assert_close(out[:, s], _fn()(c["x"][:, s], c["dt"][:, s], c["A"], c["B"][:, s], c["C"][:, s], 256, z=c["z"][:, s], **kw), TOL_BF16, f"seq {i}")
    assert _status() == 0


@pytest.mark.parametrize("name,dim", [("x", 0), ("z", 0), ("B", 2), ("C", 0), ("C", 2), ("x", 2)])
def test_expanded_inputs(name, dim):
    """A tensor expanded over the batch, the heads or the groups (stride 0), which is not for TMA, is read in place all the same."""
    inp = make(420, 2, 300, 4, 64, 2, 128, torch.bfloat16, init=True)
    c = {k: _c(v) for k, v in inp.items()}
    full = c[name].narrow(dim, 0, 1).expand(c[name].shape)
    c[name], inp[name] = full, full.cpu().contiguous()
    f = lambda t: None if t is None else t.float()
    want, wfin = oracle.ssd_chunk_scan(f(inp["x"]), f(inp["dt"]), inp["A"], f(inp["B"]), f(inp["C"]), 256, inp["D"], f(inp["z"]), inp["dt_bias"],
                                       inp["initial_states"], dt_softplus=True)
    got, fin = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], initial_states=c["initial_states"],
                     dt_softplus=True, return_final_states=True)
    assert _status() == 0
    assert_close(got, want, TOL_BF16, f"{name} expanded over {dim}: out")
    assert_close(fin, wfin, TOL_BF16, f"{name} expanded over {dim}: final states")
