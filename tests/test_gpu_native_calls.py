"""The native call path of the operators against their Python path: same results bit for bit, and calls that the native
path has to decline (tensors to convert or copy, strided rows, no-heads forms) still come out right."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


class _Declines:
    def __getattr__(self, name):
        return lambda *a: None


def both(monkeypatch, call):
    from mamba_b200 import _lib
    got = call()
    with monkeypatch.context() as m:
        m.setattr(_lib, "host", lambda: _Declines())
        want = call()
    flat = lambda r: [t for t in (r if isinstance(r, tuple) else (r,)) if t is not None]
    for a, b in zip(flat(got), flat(want), strict=True):
        assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride() and torch.equal(a, b)


def r(*s, dtype=torch.float32, seed=0):
    return torch.randn(*s, generator=torch.Generator(device=DEV).manual_seed(seed + sum(s)), device=DEV).to(dtype)


@pytest.mark.parametrize("form", ["plain", "groups", "constant_bc", "permuted", "half_params", "strided_time"])
def test_scan(monkeypatch, form):
    from mamba_b200 import selective_scan_fn
    b, d, L, N, G = 2, 64, 75, 16, 2 if form == "groups" else 1
    u, delta, z = (r(b, d, L, seed=i) for i in range(3))
    if form == "permuted":
        u, delta, z = (t.permute(1, 0, 2).contiguous().permute(1, 0, 2) for t in (u, delta, z))
    if form == "strided_time":
        u = r(b, d, 2 * L)[..., ::2]
    A, D, bias = -torch.exp(r(d, N)), r(d), r(d) - 3
    if form == "half_params":
        A, D, bias = A.half(), D.half(), bias.half()
    B, C = (r(d, N), r(d, N, seed=1)) if form == "constant_bc" else (r(b, G, N, L), r(b, N, L) if G == 1 else r(b, G, N, L, seed=1))
    both(monkeypatch, lambda: selective_scan_fn(u, delta, A, B, C, D, z, bias, delta_softplus=True, return_last_state=True))


@pytest.mark.parametrize("form", ["heads", "flat", "indices", "long_indices", "half_D"])
def test_state_update(monkeypatch, form):
    from mamba_b200 import selective_state_update
    b, H, P, N = 3, 4, 16, 32
    if form == "flat":
        args = [r(b, P, N), r(b, P), r(b, P, seed=1), -torch.exp(r(P, N)), r(b, N), r(b, N, seed=1), r(P), r(b, P, seed=2), r(P, seed=3)]
    else:
        args = [r(b, H, P, N), r(b, H, P), r(b, H, 1).expand(b, H, P), -torch.exp(r(H, 1, 1)).expand(H, P, N), r(b, 2, N), r(b, 2, N, seed=1),
                r(H, 1).expand(H, P), r(b, H, P, seed=2), r(H, 1, seed=3).expand(H, P)]
    if form == "half_D":
        args[6] = args[6].half()
    idx = torch.tensor([2, -1, 0], device=DEV, dtype=torch.int64 if form == "long_indices" else torch.int32) if "indices" in form else None

    def call():
        state = args[0].clone()
        return selective_state_update(state, *args[1:], dt_softplus=True, state_batch_indices=idx), state
    both(monkeypatch, call)


@pytest.mark.parametrize("layout", ["time", "channels", "neither"])
def test_conv_and_norm(monkeypatch, layout):
    from mamba_b200 import causal_conv1d_fn, causal_conv1d_update, rmsnorm_fn
    b, d, L = 2, 40, 29
    x = {"time": r(b, d, L), "channels": r(b, L, d).transpose(1, 2), "neither": r(b, d, 2 * L)[..., ::2].transpose(0, 1).contiguous().transpose(0, 1)}[layout]
    w, bias = r(d, 4), r(d)
    both(monkeypatch, lambda: causal_conv1d_fn(x, w, bias, activation="silu"))
    both(monkeypatch, lambda: causal_conv1d_update(x[:, :, 0], r(b, d, 4), w, bias, "silu"))
    both(monkeypatch, lambda: rmsnorm_fn(x, r(L), z=r(b, d, L, seed=5), norm_before_gate=False))


@pytest.mark.parametrize("norm,batch,ngroups,init", [(True, 1, 1, False), (True, 2, 2, True), (False, 2, 1, False)])
def test_ssd_and_block(monkeypatch, norm, batch, ngroups, init):
    from mamba_b200 import mamba_chunk_scan_combined, mamba_split_conv1d_scan_combined
    H, P, N, L = 4, 64, 128, 130
    dim, ch = H * P, H * P + 2 * ngroups * N
    zx = r(batch, L, dim + ch + H, dtype=torch.bfloat16)
    w, A, bias, D = 0.3 * r(ch, 4, dtype=torch.bfloat16), -1 - torch.rand(H, device=DEV), r(H) - 3, r(H)
    h0 = r(batch, H, P, N) if init else None
    kw = dict(initial_states=h0, return_final_states=True, headdim=P, ngroups=ngroups, norm_before_gate=False)
    if norm:
        kw.update(rmsnorm_weight=r(dim, dtype=torch.bfloat16), outproj_weight=0.1 * r(32, dim, dtype=torch.bfloat16))
    both(monkeypatch, lambda: mamba_split_conv1d_scan_combined(zx, w, None, bias, A, D, 256, **kw))
    x, B, C = r(batch, L, H, P), r(batch, L, ngroups, N), r(batch, L, ngroups, N, seed=1)
    both(monkeypatch, lambda: mamba_chunk_scan_combined(x, r(batch, L, H), A, B, C, 64, D=D.half(), z=x, dt_bias=bias, initial_states=h0,
                                                        dt_softplus=True, return_final_states=True))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("variable", [True, False])
def test_gradients_own_their_storage(dtype, variable):
    """What autograd hands on may be kept as .grad: no gradient holds the memory, or shares the version counter, of another."""
    from mamba_b200 import selective_scan_fn
    b, d, L, N = 2, 8, 300, 4
    u, delta, z = (r(b, d, L, seed=i).to(dtype).requires_grad_() for i in range(3))
    B, C = (r(b, 1, N, L, seed=i).to(dtype).requires_grad_() if variable else r(d, N, seed=i).requires_grad_() for i in range(2))
    A, D, bias = (-torch.exp(r(d, N))).requires_grad_(), r(d).requires_grad_(), (r(d) - 3).requires_grad_()
    leaves = (u, delta, A, B, C, D, z, bias)
    grads = torch.autograd.grad(selective_scan_fn(u, delta, A, B, C, D, z, bias, delta_softplus=True), leaves, r(b, d, L, seed=9).to(dtype))
    for t, g in zip(leaves, grads):
        assert g.untyped_storage().nbytes() == t.numel() * t.element_size()
    versions = [g._version for g in grads]
    grads[5].add_(1)
    assert [g._version for g in grads] == [v + (i == 5) for i, v in enumerate(versions)]
