"""16-bit SSD calls outside headdim 64 / dstate 128 / chunk 256: products as exact as fp32's.  Outputs are no further from the oracle
(which computes in double) than its own result rounded to their type, and fp32 states as close as those of fp32 inputs: 2e-5 relative, which
exponentials of differences of running sums of several hundred leave."""
import pytest
import torch

import oracle
from test_gpu_ssd import DEV, _c, _fn, _packed, _status, make

pytestmark = pytest.mark.gpu
F32 = 2e-5
DTYPES = [torch.bfloat16, torch.float16]


def rel(got, want):
    got, want = got.detach().double().cpu(), want.double()
    assert torch.isfinite(got).all()
    return ((got - want).norm() / want.norm().clamp_min(1e-30)).item()


def check_out(got, want, what):
    rounding = rel(want.to(got.dtype), want)
    assert rel(got, want) <= 1.01 * rounding + F32, f"{what}: {rel(got, want):.3e}, rounding alone {rounding:.3e}"


def run(inp, Q, what, want=None, **kw):
    f = lambda t: None if t is None else t.float()
    want, wfin = want or oracle.ssd_chunk_scan(f(inp["x"]), f(inp["dt"]), inp["A"], f(inp["B"]), f(inp["C"]), Q, inp["D"], f(inp["z"]), inp["dt_bias"],
                                               inp["initial_states"], dt_softplus=True)
    c = {k: _c(v) for k, v in inp.items()}
    got, fin = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], Q, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], initial_states=c["initial_states"],
                     dt_softplus=True, return_final_states=True, **kw)
    assert _status() == 0
    check_out(got, want, what)
    assert rel(fin, wfin) <= F32, f"{what}: final states {rel(fin, wfin):.3e}"


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("P,N,G,H,Q,L", [(64, 64, 1, 6, 256, 300), (128, 128, 2, 4, 256, 257), (64, 128, 1, 3, 128, 385), (40, 24, 1, 5, 64, 129), (8, 8, 2, 2, 32, 70),
                                         (72, 136, 1, 2, 256, 128), (7, 200, 1, 2, 100, 250), (65, 65, 1, 2, 63, 127), (64, 64, 1, 2, 1024, 1300), (64, 256, 1, 2, 256, 1)])
def test_shapes(dtype, P, N, G, H, Q, L):
    run(make(700 + P + N, 2, L, H, P, G, N, dtype, has_z=L % 2 == 0, D_hdim=P % 2 == 0, init=True), Q, f"P{P} N{N} Q{Q} L{L}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("step", [1, 3, 8])
def test_rows_inside_wider_buffers(dtype, step):
    """Rows off 16-byte boundaries, and tensors expanded over the heads or groups."""
    inp = make(720, 2, 200, 4, 64, 2, 64, dtype, init=True)

    def wide(t):
        buf = torch.full(t.shape[:-1] + (t.shape[-1] + step,), float("nan"), dtype=dtype)
        buf[..., step:] = t
        return buf.to(DEV)[..., step:]

    ref = dict(inp)
    for k in ("x", "B", "C", "z"):
        ref[k] = inp[k]
        inp[k] = wide(inp[k])
    f = lambda t: t.float()
    run(inp, 128, f"step {step}", oracle.ssd_chunk_scan(f(ref["x"]), f(ref["dt"]), ref["A"], f(ref["B"]), f(ref["C"]), 128, ref["D"], f(ref["z"]), ref["dt_bias"],
                                                        ref["initial_states"], dt_softplus=True))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("P,N,H,Q,lens", [(64, 64, 4, 256, [100, 156, 1, 300, 40]), (128, 128, 2, 128, [257, 255, 130]), (40, 24, 2, 64, [3, 128, 200]),
                                          (64, 128, 2, 256, [40, 1, 100, 50, 65])])       # the last within a chunk: nothing of it in 16 bits
def test_packed(dtype, P, N, H, Q, lens):
    inp, seq_idx, cu = _packed(740 + N, lens, H, P, 1, N, dtype)
    c = {k: _c(v) for k, v in inp.items()}
    out, fin, var = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], Q, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], seq_idx=seq_idx.to(DEV), cu_seqlens=cu.to(DEV),
                          dt_softplus=True, return_final_states=True, return_varlen_states=True)
    assert _status() == 0
    f = lambda t: t.float()
    for i in range(len(lens)):
        sl = slice(int(cu[i]), int(cu[i + 1]))
        want, wfin = oracle.ssd_chunk_scan(f(inp["x"][:, sl]), f(inp["dt"][:, sl]), inp["A"], f(inp["B"][:, sl]), f(inp["C"][:, sl]), Q, inp["D"],
                                           f(inp["z"][:, sl]), inp["dt_bias"], None, dt_softplus=True)
        if N != 128 or P != 64:
            check_out(out[:, sl], want, f"packed out seq {i}")
        assert rel(var[i:i + 1], wfin) <= F32, f"end state of sequence {i}: {rel(var[i:i + 1], wfin):.3e}"


def test_half_precision_keeps_the_range_of_fp32():
    """C.B and states beyond 65504, the largest half, with outputs that fit it again."""
    inp = make(760, 1, 200, 2, 64, 1, 64, torch.float16, has_z=False, init=True)
    inp["B"], inp["C"], inp["x"] = inp["B"] * 200, inp["C"] * 200, inp["x"] * 1e-3
    inp["initial_states"] = inp["initial_states"] * 1e5
    inp["C"][:, :100] *= 1e-4
    inp["C"][:, 100:] *= 0.03
    assert (torch.einsum("blgn,bkgn->blk", inp["C"].float(), inp["B"].float()).abs().max() > 65504 / 4)
    run(inp, 128, "large")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("N", [64, 128])
def test_infinities_stay_in_their_sequence(dtype, N):
    """A packed sequence with infinite and NaN inputs: the end states of the others are what they were, its own is not finite."""
    lens = [60, 70, 50]
    inp, seq_idx, cu = _packed(780 + N, lens, 2, 64, 1, N, dtype)

    def end_states():
        c = {k: _c(v) for k, v in inp.items()}
        return _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, D=c["D"], dt_bias=c["dt_bias"], seq_idx=seq_idx.to(DEV), cu_seqlens=cu.to(DEV),
                     dt_softplus=True, return_varlen_states=True)[1].cpu()
    before = end_states()
    inp["B"][0, 70, 0, 3] = float("inf")
    inp["x"][0, 80, 1, 5] = float("nan")
    after = end_states()
    assert torch.equal(after[0], before[0]) and torch.equal(after[2], before[2])
    assert torch.isinf(after[1, 0, :, 3]).all() and torch.isnan(after[1, 1, 5]).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["x", "C"])
def test_infinite_inputs_give_infinite_outputs(dtype, name):
    """An infinity is one in every output it reaches through nonzero factors, not a NaN, and reaches no earlier block of 128 rows."""
    inp = make(790, 1, 300, 2, 64, 1, 64, dtype, has_z=False, init=True)
    t = 140
    inp[name][0, t, 0, 9] = float("inf")
    c = {k: _c(v) for k, v in inp.items()}
    run_it = lambda: _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, dt_bias=c["dt_bias"], initial_states=c["initial_states"], dt_softplus=True).cpu()
    out = run_it()
    assert torch.isfinite(out[0, :128]).all()
    if name == "x":
        assert torch.isinf(out[0, t:t + 20, 0, 9]).all() and torch.isfinite(out[0, :, 1]).all()
    else:
        assert not torch.isfinite(out[0, t]).any() and torch.isfinite(out[0, 128:t]).all() and torch.isfinite(out[0, t + 1:]).all()
