"""The split-product stages where their short cuts end: decays that cannot be factorised over 32 steps (steeper than 2^100, or rising),
fp32 inputs at the edges of tiles, and fp32 infinities and NaNs, which the tensor core leaves to fp32 FMAs."""
import math

import pytest
import torch

import oracle
from test_gpu_ssd import DEV, _c, _fn, _packed, make
from test_gpu_ssd_split import F32, check_out, rel, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("A", [-400.0, -40.0])
def test_decays_formed_one_by_one(dtype, A):
    """One head with decays of that kind among ordinary ones; 32 steps of the steepest take it past the smallest fp32."""
    inp = make(900, 2, 300, 3, 64, 1, 64, dtype, init=True)
    inp["A"][1] = A
    run(inp, 256, f"A {A}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_rising_sums(dtype):
    """A > 0: differences of the running sums are cut off at 0, as documented, so that no decay exceeds 1."""
    inp = make(905, 1, 200, 2, 64, 1, 64, dtype, has_z=False, init=True)
    inp["A"][1] = 0.02
    d = {k: v.double() for k, v in inp.items() if v is not None}
    dt = torch.nn.functional.softplus(d["dt"] + d["dt_bias"])[0]                          # (L, H)
    sums = torch.cumsum(dt * d["A"], 0).T                                                 # (H, L)
    decay = torch.exp((sums[:, :, None] - sums[:, None, :]).clamp(max=0)).tril() * dt.T[:, None, :]
    want = torch.einsum("mn,kn,hmk,khp->mhp", d["C"][0, :, 0], d["B"][0, :, 0], decay, d["x"][0])
    want += torch.einsum("mn,hm,hpn->mhp", d["C"][0, :, 0], torch.exp(sums), d["initial_states"][0]) + d["x"][0] * (d["D"] if d["D"].dim() == 2 else d["D"][:, None])
    wfin = torch.exp(sums[:, -1])[:, None, None] * d["initial_states"][0] + torch.einsum("kn,hk,khp->hpn", d["B"][0, :, 0], decay[:, -1], d["x"][0])
    run(inp, 256, "rising", (want[None].float(), wfin[None].float()))


def _steady(inp, step):
    """Every step has length 0.1375 and decays its head by `step` nats, with no skip that would cover the sums."""
    inp["A"][:], inp["dt"][:], inp["D"] = -step / 0.1375, 0.0, None
    inp["dt_bias"][:] = math.log(math.expm1(0.1375))
    return inp


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("P", [64, 128])
def test_steep_decays_and_small_products(dtype, P):
    """98 powers of two within 32 steps, the steepest that is factorised: C.B of 1e-15 meets column factors of 2^-98, whose product would be subnormal."""
    inp = _steady(make(960 + P, 2, 300, 3, P, 1, 64, dtype, has_z=False), 2.2)
    inp["B"], inp["C"] = inp["B"] * 1e-8, inp["C"] * 1e-8
    run(inp, 256, f"small products P{P}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_steep_decays_and_a_step_of_almost_no_length(dtype):
    """The only step with an input has dt of 1e-15 and 30 of the steepest steps behind it in its range: the column factor would be subnormal."""
    inp = _steady(make(962, 1, 200, 2, 64, 1, 64, dtype, has_z=False), 2.2)
    inp["dt"][:, 33] = -34.5 - inp["dt_bias"]
    keep = torch.arange(200) == 33
    inp["x"][:, ~keep] = 0
    run(inp, 256, "short step")


def test_weights_within_32_steps():
    """dt and dt exp(-1.4) for the step itself and the next, though the chunk's sums reach 358, where they are rounded to 3e-5.  Inputs 65 steps
    apart, so that what came before has decayed to nothing."""
    L, decay = 65 * 128, 1.4
    inp = _steady(make(964, 1, L, 2, 64, 1, 64, torch.float32, has_z=False), decay)
    inp["B"][:], inp["C"][:], inp["x"][:] = 0.0, 0.0, 0.0
    inp["B"][..., 0], inp["C"][..., 0] = 1.0, 1.0
    at = torch.arange(0, L, 65)
    inp["x"][:, at] = 1.0
    dt = torch.full_like(inp["dt"], 0.1375)
    out = _fn()(*(_c(t) for t in (inp["x"], dt, inp["A"], inp["B"], inp["C"])), 256).cpu().double()
    dt = dt.double()[0, 0, :, None]
    rounding = 4 * 2.0 ** -23 + 4 * 2.0 ** -24                                   # two exponentials of at most 2 ulp, four roundings
    assert (out[:, at] / dt - 1).abs().max() <= rounding
    at = at[at % 32 != 31]                                                       # (the next step belongs to the same 32)
    # two distances of up to 31 steps, summed in five rounds of 2, 4, 8, 16 and 31, then times log2 e: each rounds by at most 2^-24 of its size
    assert (out[:, at + 1] / (dt * torch.exp(dt * inp["A"].double()[:, None])) - 1).abs().max() <= rounding + 2 * 2.0 ** -24 * (61 + 31) * decay


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("packed", [False, True])
def test_weights_of_end_states(dtype, packed):
    """The only input of a sequence is the last but one: its end state is dt exp(-1.4) x B, though the chunk's sums reach 350, where they are rounded to 3e-5."""
    lens = [67, 130, 250, 256, 40, 31, 301, 93] if packed else [245]
    inp = _steady(make(974, 1, sum(lens), 2, 64, 1, 64, dtype, has_z=False), 1.4)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    dt, A = torch.full_like(inp["dt"], 0.125), torch.full_like(inp["A"], -11.2)
    at = cu[1:].long() - 2
    keep = torch.zeros(sum(lens), dtype=torch.bool).index_fill(0, at, True)
    inp["x"][:, ~keep] = 0
    kw = dict(return_final_states=True)
    if packed:
        seq = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens))[None].to(torch.int32)
        kw.update(seq_idx=seq.to(DEV), cu_seqlens=cu.to(DEV), return_varlen_states=True)
    got = _fn()(*(_c(t) for t in (inp["x"], dt, A, inp["B"], inp["C"])), 256, **kw)[-1].cpu().double()
    step = dt.double()[0, 0, 0] * A.double()[0]
    want = dt.double()[0, 0, 0] * torch.exp(step) * torch.einsum("shp,sn->shpn", inp["x"][0, at].double(), inp["B"][0, at, 0].double())
    same = (at % 256) % 32 != 31                                    # (in the 32 steps of the last one)
    # the exponential: 2 ulp and 2^-24 of its argument; the weight, the weighted x, their cut and the sum: a rounding each; truncation: 2^-23
    bound = (2 * 2 + 1.4 + 4 + 2) * 2.0 ** -24
    assert same.any() and ((got - want).abs() <= bound * want.abs())[same].all()


@pytest.mark.parametrize("x,B,C", [(1e-36, 1, 1), (1, 1e-36, 1), (1, 1, 1e-36), (1e20, 1e12, 1e-3), (1e-20, 1e15, 1e15), (1e37, 1e-10, 1e-20), (1e-20, 1e37, 1e-10), (1e-10, 1e-20, 1e37)])
def test_fp32_keeps_its_range(x, B, C):
    """Operands near the smallest normal number have all their bits, and operands and sums too large for the tensor core's are what fp32 holds."""
    inp = make(976, 2, 300, 3, 64, 1, 64, torch.float32, has_z=False, init=True)
    want, wfin = oracle.ssd_chunk_scan(inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], 256, None, None, inp["dt_bias"], inp["initial_states"], dt_softplus=True)
    inp["x"], inp["B"], inp["C"], inp["initial_states"] = inp["x"] * x, inp["B"] * B, inp["C"] * C, inp["initial_states"] * (x * B)
    c = {k: _c(v) for k, v in inp.items()}
    out, fin = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, dt_bias=c["dt_bias"], initial_states=c["initial_states"], dt_softplus=True, return_final_states=True)
    assert rel(out.double() / (x * B * C), want) <= F32 and rel(fin.double() / (x * B), wfin) <= F32


@pytest.mark.parametrize("seed", [970, 971, 972])
def test_fp32_sums_without_decay(seed):
    """Next to no decay, so that the sums over 256 steps and over the states are the whole error.  FMAs one after the other round each of n sums
    that grow as their square root by 0.29 ulp: 0.29 2^-23 sqrt(256 / 2) = 3.9e-7 for the states, of which 3.3e-7 was measured, and 4.3e-7 for
    the outputs.  Sums left to the tensor core, which cuts off where FMAs round, were at 4.0e-7 and 6.4e-7."""
    inp = make(seed, 2, 1500, 8, 64, 1, 64, torch.float32, has_z=False)
    inp["A"] *= 1e-4
    want, wfin = oracle.ssd_chunk_scan(inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], 256, inp["D"], None, inp["dt_bias"], None, dt_softplus=True)
    c = {k: _c(v) for k, v in inp.items()}
    got, fin = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, D=c["D"], dt_bias=c["dt_bias"], dt_softplus=True, return_final_states=True)
    assert rel(fin, wfin) <= 3.3e-7 and rel(got, want) <= 4.3e-7, (rel(fin, wfin), rel(got, want))


@pytest.mark.parametrize("P,N,H,Q,L", [(64, 64, 2, 256, 129), (128, 128, 1, 128, 257), (65, 66, 2, 64, 65), (7, 130, 1, 100, 101), (64, 64, 1, 1024, 1100), (1, 1, 1, 1, 3)])
def test_fp32_shapes(P, N, H, Q, L):
    run(make(910 + P + N, 2, L, H, P, 1, N, torch.float32, has_z=L % 2 == 0, D_hdim=P % 2 == 0, init=True), Q, f"P{P} N{N} Q{Q} L{L}")


def test_fp32_gate_far_below_zero():
    """silu(z) for z below -87.3, where 1 + exp(-z) exceeds 2^126: -1e-36 and not zero (below -88.7 exp(-z) is infinite, as in silu itself)."""
    inp = make(966, 1, 130, 2, 64, 1, 64, torch.float32)
    inp["z"] = torch.linspace(-88.7, -80.0, inp["z"].numel()).reshape(inp["z"].shape)
    c = {k: _c(v) for k, v in inp.items()}
    out = lambda z: _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 128, D=c["D"], z=z, dt_bias=c["dt_bias"], dt_softplus=True).cpu().double()
    z = inp["z"].double()
    want = out(None) * z * torch.sigmoid(z)
    keep = want.abs() > 1.2e-38                                              # (what is subnormal has fewer bits)
    assert (keep & (z < -87.4)).any() and ((out(c["z"]) - want).abs()[keep] / want.abs()[keep]).max() <= 1e-6       # five roundings and expf's


@pytest.mark.parametrize("name", ["x", "B", "C"])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38])
def test_fp32_values_that_cannot_be_cut(name, value):
    """They reach what they reach through nonzero factors, as infinities or NaNs, and leave everything else as exact as it was."""
    t, e = 140, 9
    inp = make(920, 1, 300, 2, 64, 1, 64, torch.float32, has_z=False, init=True)
    kw = dict(dt_softplus=True)
    want, wfin = oracle.ssd_chunk_scan(inp["x"], inp["dt"], inp["A"], inp["B"], inp["C"], 256, inp["D"], None, inp["dt_bias"], inp["initial_states"], **kw)
    inp[name][0, t, 0, e] = value
    c = {k: _c(v) for k, v in inp.items()}
    out, fin = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, D=c["D"], dt_bias=c["dt_bias"], initial_states=c["initial_states"], return_final_states=True, **kw)
    out, fin = out.cpu(), fin.cpu()
    assert rel(out[0, :t], want[0, :t]) <= F32                               # nothing goes back in time
    if name == "x":                                                          # one column of one head
        assert torch.isfinite(out[0, :, 1]).all() and rel(out[0, :, 1], want[0, :, 1]) <= F32
        keep = torch.arange(64) != e
        assert rel(out[0, :, 0, keep], want[0, :, 0, keep]) <= F32 and rel(fin[0, 0, keep], wfin[0, 0, keep]) <= F32
        if value != 3.4e38:
            assert not torch.isfinite(out[0, t, 0, e])
    if name == "B":                                                          # one state of every head
        keep = torch.arange(64) != e
        assert rel(fin[..., keep], wfin[..., keep]) <= F32
        if value != 3.4e38:                                                  # (times a decay of 0 a NaN)
            assert not torch.isfinite(fin[..., e]).any() and not torch.isfinite(out[0, t]).any()
    if name == "C":                                                          # one step
        later = torch.arange(300) != t
        assert rel(out[0, later], want[0, later]) <= F32 and rel(fin, wfin) <= F32
        if value != 3.4e38:
            assert not torch.isfinite(out[0, t]).any()


@pytest.mark.parametrize("name", ["x", "B", "C"])
@pytest.mark.parametrize("P,N,lens", [(64, 64, [100, 200]), (72, 40, [100, 199]), (136, 130, [3, 250])])
def test_fp32_values_too_large_to_be_cut(name, P, N, lens):
    """The tiles that hold one are added with fp32 FMAs: gated, with D per column, packed and ragged, all is what the oracle gives."""
    t, e = sum(lens) - 160, 9
    inp, seq_idx, cu = _packed(925 + P, lens, 3, P, 1, N, torch.float32)
    inp["D"] = torch.randn(3, P, generator=torch.Generator().manual_seed(P))
    inp[name][0, t, 0, e] = 3e36
    c = {k: _c(v) for k, v in inp.items()}
    out, _, var = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 128, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], seq_idx=seq_idx.to(DEV), cu_seqlens=cu.to(DEV),
                        dt_softplus=True, return_final_states=True, return_varlen_states=True)
    out, var = out.cpu(), var.cpu()
    for i in range(2):
        sl = slice(int(cu[i]), int(cu[i + 1]))
        want, wfin = oracle.ssd_chunk_scan(inp["x"][:, sl], inp["dt"][:, sl], inp["A"], inp["B"][:, sl], inp["C"][:, sl], 128, inp["D"], inp["z"][:, sl], inp["dt_bias"], None,
                                           dt_softplus=True)
        got, state, at = out[:, sl], var[i:i + 1], max(t - sl.start, 0) if i == 1 else sl.stop
        assert rel(got[:, :at], want[:, :at]) <= F32 or at == 0
        if i == 0 or name == "C":
            assert rel(state, wfin) <= F32
        if i == 0:
            continue
        assert rel(got[:, at], want[:, at]) <= F32
        if name == "x":                                                      # one column of one head
            cols = torch.arange(P) != e
            assert rel(got[:, :, 0, cols], want[:, :, 0, cols]) <= F32 and rel(got[:, :, 1:], want[:, :, 1:]) <= F32
            assert rel(state[:, 0, cols], wfin[:, 0, cols]) <= F32 and rel(state[:, 1:], wfin[:, 1:]) <= F32 and rel(state[:, 0, e], wfin[:, 0, e]) <= F32
        if name == "B":                                                      # one state of every head
            keep = torch.arange(N) != e
            assert rel(state[..., keep], wfin[..., keep]) <= F32 and rel(state[..., e], wfin[..., e]) <= F32
        if name == "C":                                                      # one step
            assert rel(got[:, at + 1:], want[:, at + 1:]) <= F32


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("P,N,L", [(64, 64, 300), (72, 40, 299), (136, 130, 255)])
def test_gate_and_skip_where_a_tile_is_left_out(dtype, P, N, L):
    """16 bits: what an infinity in one column does not reach is gated and has its D as everywhere."""
    t, e = 140, 9
    inp = make(927 + P, 1, L, 3, P, 1, N, dtype, D_hdim=True, init=True)
    f = lambda v: v.float()
    want, _ = oracle.ssd_chunk_scan(f(inp["x"]), f(inp["dt"]), inp["A"], f(inp["B"]), f(inp["C"]), 128, inp["D"], f(inp["z"]), inp["dt_bias"], inp["initial_states"], dt_softplus=True)
    inp["x"][0, t, 1, e] = float("inf")
    c = {k: _c(v) for k, v in inp.items()}
    out = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 128, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], initial_states=c["initial_states"], dt_softplus=True).cpu()
    keep = torch.arange(P) != e
    check_out(out[0, :t], want[0, :t], "earlier steps")
    check_out(out[0, :, 0], want[0, :, 0], "other head")
    check_out(out[0, :, 1, keep], want[0, :, 1, keep], "other columns")
    assert not torch.isfinite(out[0, t, 1, e])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("P,N,G,H", [(64, 64, 1, 15), (72, 40, 3, 15), (64, 136, 1, 9)])
def test_two_heads_share_their_b(dtype, P, N, G, H):
    """Enough chunks and heads for the chunk states to go by pairs, an odd head or column tile out among them."""
    run(make(930 + P + N, 2, 1000, H, P, G, N, dtype, has_z=False, init=True), 64, f"P{P} N{N} G{G} H{H}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("P,N,H,L", [(128, 64, 8, 1000), (72, 40, 9, 999), (200, 130, 5, 1000)])
def test_two_column_tiles_share_their_a(dtype, P, N, H, L):
    """Enough chunks and heads for the outputs to go by two column tiles of a head, the second (third) of them ragged."""
    run(make(940 + P + N, 2, L, H, P, 1, N, dtype, has_z=P == 72, D_hdim=P == 200, init=True), 64, f"P{P} N{N} H{H}")


# two heads of a group share B (U2: 64 columns, enough heads and chunks), or two column tiles of a head share A (W2: more columns)
U2 = [(torch.float32, 64, 64, 15), (torch.float16, 64, 64, 15), (torch.float16, 72, 40, 9)]
W2 = [(torch.bfloat16, 128, 64, 8), (torch.float16, 128, 64, 8), (torch.float16, 200, 130, 5)]


@pytest.mark.parametrize("dtype,P,N,H", U2 + W2)
def test_shared_operands_in_packed_sequences(dtype, P, N, H):
    lens = [100, 156, 1, 300, 43, 64, 640, 63, 65, 568]
    inp, seq_idx, cu = _packed(980 + P + N, lens, H, P, 1, N, dtype)
    c = {k: _c(v) for k, v in inp.items()}
    out, fin, var = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 64, D=c["D"], z=c["z"], dt_bias=c["dt_bias"], seq_idx=seq_idx.to(DEV), cu_seqlens=cu.to(DEV),
                          dt_softplus=True, return_final_states=True, return_varlen_states=True)
    f = lambda t: t.float()
    for i in range(len(lens)):
        sl = slice(int(cu[i]), int(cu[i + 1]))
        want, wfin = oracle.ssd_chunk_scan(f(inp["x"][:, sl]), f(inp["dt"][:, sl]), inp["A"], f(inp["B"][:, sl]), f(inp["C"][:, sl]), 64, inp["D"], f(inp["z"][:, sl]),
                                           inp["dt_bias"], None, dt_softplus=True)
        check_out(out[:, sl], want, f"packed out seq {i}")
        assert rel(var[i:i + 1], wfin) <= F32, f"end state of sequence {i}: {rel(var[i:i + 1], wfin):.3e}"
    assert rel(fin, wfin) <= F32


@pytest.mark.parametrize("dtype,P,N,H", U2 + W2)
@pytest.mark.parametrize("name", ["x", "B"])
def test_shared_operands_with_an_infinity(dtype, P, N, H, name):
    """In the second of two heads, and in the second column tile where there is one: it stays in what it reaches."""
    t, e = 140, P - 1 if name == "x" else 9
    inp = make(990 + P + N, 2, 1000, H, P, 1, N, dtype, has_z=False, init=True)
    f = lambda v: v.float()
    want, wfin = oracle.ssd_chunk_scan(f(inp["x"]), f(inp["dt"]), inp["A"], f(inp["B"]), f(inp["C"]), 64, inp["D"], None, inp["dt_bias"], inp["initial_states"], dt_softplus=True)
    inp[name][0, t, 1 if name == "x" else 0, e] = float("inf")
    c = {k: _c(v) for k, v in inp.items()}
    out, fin = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 64, D=c["D"], dt_bias=c["dt_bias"], initial_states=c["initial_states"], dt_softplus=True,
                     return_final_states=True)
    out, fin = out.cpu(), fin.cpu()
    check_out(out[1], want[1], "other row")
    check_out(out[0, :t], want[0, :t], "earlier steps")
    assert rel(fin[1], wfin[1]) <= F32
    if name == "x":
        others, keep = torch.arange(H) != 1, torch.arange(P) != e
        check_out(out[0, :, others], want[0, :, others], "other heads")
        check_out(out[0, :, 1, keep], want[0, :, 1, keep], "other columns")
        assert torch.isinf(out[0, t, 1, e]) and rel(fin[0, others], wfin[0, others]) <= F32 and rel(fin[0, 1, keep], wfin[0, 1, keep]) <= F32
    else:
        keep = torch.arange(N) != e
        assert not torch.isfinite(out[0, t]).any() and rel(fin[0][..., keep], wfin[0][..., keep]) <= F32


@pytest.mark.parametrize("dtype,P,N,H", U2 + W2)
def test_shared_operands_and_decays_formed_one_by_one(dtype, P, N, H):
    inp = make(1000 + P + N, 2, 1000, H, P, 1, N, dtype, has_z=False, init=True)
    inp["A"][1], inp["A"][3] = -400.0, -40.0
    run(inp, 64, f"steep P{P} N{N}")


def test_end_states_of_many_short_sequences():
    """Enough sequences and heads for the 64-row tiles of the end states; lengths around 64, 128 and 256, one across two chunks."""
    lens = [1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300] + [5] * 39
    inp, seq_idx, cu = _packed(950, lens, 24, 64, 1, 128, torch.bfloat16)
    c = {k: _c(v) for k, v in inp.items()}
    _, _, var = _fn()(c["x"], c["dt"], c["A"], c["B"], c["C"], 256, D=c["D"], dt_bias=c["dt_bias"], seq_idx=seq_idx.to(DEV), cu_seqlens=cu.to(DEV),
                      dt_softplus=True, return_final_states=True, return_varlen_states=True)
    for i in range(len(lens)):
        sl = slice(int(cu[i]), int(cu[i + 1]))
        _, wfin = oracle.ssd_chunk_scan(inp["x"][:, sl].float(), inp["dt"][:, sl].float(), inp["A"], inp["B"][:, sl].float(), inp["C"][:, sl].float(), 256, inp["D"], None,
                                        inp["dt_bias"], None, dt_softplus=True)
        inside = int(cu[i]) // 256 == (int(cu[i + 1]) - 1) // 256        # nothing of it went through a 16-bit state
        assert rel(var[i:i + 1], wfin) <= (F32 if inside else 3e-3), f"end state of sequence {i}: {rel(var[i:i + 1], wfin):.3e}"
