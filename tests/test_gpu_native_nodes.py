"""The native autograd nodes against the torch.autograd.Function classes behind them, over the forms that both accept: the same
library calls on the same values, so results are compared bit for bit.  And what neither takes is still refused."""
import pytest
import torch

from semicat_b200 import _lib, _nodes, dual_ops, functional, ops, rotary, safe_sdpa_jvp, sdpa_jvp, set_kernel_family

pytestmark = pytest.mark.gpu


def _rand(seed, *shape, dtype=torch.bfloat16, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _both_ways(monkeypatch, f):
    """``f()`` through the native nodes (which must take every call) and through the classes."""
    refused = []

    def strict(*a):
        out = _nodes.native(*a)
        if out is None and (a[0] != "linear" or torch.autograd.forward_ad.unpack_dual(a[1]).tangent is not None):
            refused.append(a[0])  # (a linear layer without a tangent is torch's own)
        return out

    for way in (strict, lambda *a: None):
        for m in (functional, dual_ops, rotary):
            monkeypatch.setattr(m, "native", way)
        yield f()
    assert not refused


def _equal(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.shape == y.shape and x.dtype == y.dtype and x.stride() == y.stride() and torch.equal(x, y)


def _bhsd(t, form):
    """(B, H, S, D) values in one of the memory orders that callers have them in."""
    B, H, S, D = t.shape
    if form == "bshd":
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    if form == "qkv":  # a slice of a projection
        return torch.stack((t, t, t), 2).permute(0, 3, 2, 1, 4).contiguous()[:, :, 1].transpose(1, 2)
    if form == "channels":  # not the unit stride
        return t.transpose(2, 3).contiguous().transpose(2, 3)
    if form == "expanded":
        return t[:, :1].expand(B, H, S, D)
    return t.contiguous()


@pytest.mark.parametrize("B,H,Lq,Lk,D,dtype", [(2, 3, 64, 64, 64, torch.bfloat16), (1, 2, 77, 130, 64, torch.float16), (2, 2, 130, 33, 128, torch.bfloat16),
                                               (3, 2, 129, 129, 40, torch.bfloat16), (1, 2, 33, 65, 48, torch.float16), (1, 1, 1, 1, 17, torch.bfloat16)])
@pytest.mark.parametrize("form", ["bhsd", "bshd", "qkv", "channels", "expanded"])
def test_attention(monkeypatch, B, H, Lq, Lk, D, dtype, form):
    base = [_bhsd(_rand(i, B, H, L, D, dtype=dtype, scale=0.5), form).detach() for i, L in enumerate((Lq, Lk, Lk, Lq, Lk, Lk))]
    for entry, missing, which in [(e, m, w) for e in (sdpa_jvp, safe_sdpa_jvp) for m, w in
                                  (((), "both"), ((), "tangent"), ((), "primal"), ((1,), "both"), ((0, 2), "tangent"), ((0, 1, 2), "primal"))]:
        x = [(t if entry is sdpa_jvp else t.transpose(1, 2)).detach().requires_grad_(True) for t in base]
        tang = [None if i in missing else t for i, t in enumerate(x[3:])] if len(missing) < 3 else []
        leaves = [t for t in tang if t is not None]

        def run():
            live = [i for i in range(3) if i not in missing]
            if not leaves:
                y = entry(*x[:3])
                return [y.detach(), *torch.autograd.grad(y, x[:3], _rand(9, *y.shape, dtype=dtype))]
            f = lambda *a: entry(*[a[live.index(i)] if i in live else x[i] for i in range(3)])
            y, ty = torch.func.jvp(f, tuple(x[i] for i in live), tuple(leaves))
            outs = {"both": [y, ty], "tangent": [ty], "primal": [y]}[which]
            grads = torch.autograd.grad(outs, [*x[:3], *leaves], [_rand(9 + i, *o.shape, dtype=dtype) for i, o in enumerate(outs)], allow_unused=True)
            with torch.no_grad():
                again = entry(*x[:3])
            return [y.detach(), ty.detach(), again, *grads]

        a, b = _both_ways(monkeypatch, run)
        _equal(a, b)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,S,C,dtype", [(3, 5, 256, torch.bfloat16), (2, 50, 768, torch.bfloat16), (2, 9, 512, torch.float32)])
@pytest.mark.parametrize("missing", [(), (0,), (1, 2), (0, 1, 2, 3, 4, 5)])
def test_pointwise_chain(monkeypatch, B, S, C, dtype, missing):
    H = C // 64
    norm = torch.nn.LayerNorm(C, device="cuda", bias=C != 512)
    with torch.no_grad():
        norm.weight.normal_()
    lin = torch.nn.Linear(C, 24, device="cuda", bias=C != 512).to(dtype)
    cos, sin = _rand(1, S, 32, dtype=torch.float32), _rand(2, S, 32, dtype=torch.float32)
    mod = lambda seed: _rand(seed, B, 1, 3 * C, dtype=dtype).chunk(3, dim=2)
    x0, tx0 = (_rand(s, B, S, C, dtype=dtype) for s in (3, 4))
    prim0 = [x0, *mod(5), _rand(6, B, S, C, dtype=dtype).transpose(0, 1).contiguous().transpose(0, 1), _rand(7, B, S, 3, H, 64, dtype=dtype)]
    tang0 = [tx0, *mod(8), _rand(9, B, S, C, dtype=dtype), _rand(10, B, S, 3, H, 64, dtype=dtype)]

    def chain(x, shift, scale, gate, branch, qkv):
        h = dual_ops.ln_modulate(x, norm, shift, scale[:, 0])
        h2 = dual_ops.ln_modulate(h, norm, shift[:, 0], scale, exact=True)
        z = dual_ops.gated_residual(h2, branch, gate, 0.3, True)
        z = dual_ops.gated_residual(z, branch, gate[:, 0])
        a = dual_ops.gelu_tanh(z)
        return (h, z, a, dual_ops.linear(a, lin.weight, lin.bias), *rotary.rotary_qkv(qkv, cos, sin, dtype),
                *rotary.rotary_qkv(qkv, cos, sin, torch.float32))

    def run():
        torch.manual_seed(3)
        prim = [t.detach().requires_grad_(True) for t in prim0]
        tang = [t.detach().requires_grad_(True) for t in tang0]
        leaves = [*prim, *tang, *norm.parameters(), *lin.parameters()]
        live = [i for i in range(6) if i not in missing]
        f = lambda *a: chain(*[a[live.index(i)] if i in live else prim[i] for i in range(6)])
        out = []
        for which in ("both", "tangent", "primal"):
            with dual_ops.dropout_seed(x0.device):
                if live:
                    ys, tys = torch.func.jvp(f, tuple(prim[i] for i in live), tuple(tang[i] for i in live))
                else:
                    ys, tys = chain(*prim), ()
            tys = [t for t in tys if t.requires_grad]
            outs = [*ys] if which == "primal" or not live else [*tys] if which == "tangent" else [*ys, *tys]
            cots = [_rand(50 + i, *o.shape, dtype=o.dtype) for i, o in enumerate(outs)]
            out += [*(t.detach() for t in (*ys, *tys)), *torch.autograd.grad(outs, leaves, cots, allow_unused=True)]
            with torch.no_grad():
                out += chain(*prim) if which == "primal" and not live else []
        return out

    a, b = _both_ways(monkeypatch, run)
    assert len(a) == len(b)
    for i, (p, q) in enumerate(zip(a, b)):
        assert (p is None) == (q is None), i
        if p is not None:
            # column sums are added by atomics in any order: fp32 rounding, which may flip a last bit of the 16-bit gradient
            assert p.shape == q.shape and p.dtype == q.dtype and torch.allclose(p.float(), q.float(), rtol=2 ** -7, atol=1e-4 * float(q.abs().max())), i
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,S,C,dtype", [(3, 5, 256, torch.bfloat16), (2, 50, 768, torch.bfloat16), (2, 9, 512, torch.float32), (1, 1, 1024, torch.bfloat16)])
@pytest.mark.parametrize("bias", [True, False])
def test_gated_residual_and_layer_norm_in_one(B, S, C, dtype, bias):
    """Against the two kernels: z bit for bit, the LayerNorm up to the order of its factors (one rounding of the result)."""
    norm = torch.nn.LayerNorm(C, device="cuda", bias=bias)
    with torch.no_grad():
        norm.weight.normal_()
    mod = _rand(5, B, 3 * C, dtype=dtype)
    gate, shift, scale = mod[:, :C], mod[:, C:2 * C], mod[:, 2 * C:]
    x, y = _rand(1, B, S, C, dtype=dtype), _rand(2, S, B, C, dtype=dtype).transpose(0, 1)
    with torch.no_grad():
        before = _lib.launch_count()
        z, h = dual_ops.gated_residual_ln(x, y, gate, norm, shift, scale)
        assert _lib.launch_count() - before == 1
    z2 = dual_ops.gated_residual(x, y, gate)
    h2 = dual_ops.ln_modulate(z2, norm, shift, scale)
    assert torch.equal(z, z2) and torch.allclose(h.float(), h2.float(), rtol=2 ** -7 if dtype == torch.bfloat16 else 1e-5, atol=1e-5)
    a = dual_ops.gated_residual_ln(x.requires_grad_(True), y, gate, norm, shift, scale)  # recorded: the two nodes
    assert a[0].requires_grad and torch.equal(a[0], z2) and torch.equal(a[1], h2)
    assert _lib.device_status() == 0


def _leaves(seed=0, D=64):
    return [_rand(seed + i, 2, 3, 64, D, scale=0.5).requires_grad_(True) for i in range(6)]


def test_what_is_recorded_and_refused():
    x = _leaves()
    jvp = lambda: torch.func.jvp(sdpa_jvp, tuple(x[:3]), tuple(x[3:]))
    y, ty = jvp()

    def node(t):  # behind the aliases that leaving the transform makes
        f = t.grad_fn
        while f.name().startswith("Alias"):
            f = f.next_functions[0][0]
        return f

    assert "AttentionPair" in node(y).name() and node(y) == node(ty)
    # a second reverse pass is refused, also with the cotangent a leaf
    g = torch.ones_like(ty).requires_grad_(True)
    (dq,) = torch.autograd.grad(ty, x[0], g, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        dq.float().sum().backward()
    # saved tensors go through the hooks of the forward
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.clone())[1], lambda t: t):
        y2, ty2 = jvp()
    assert len(packed) == 10
    want = torch.autograd.grad([y, ty], x, [torch.ones_like(y)] * 2)
    _equal(want, torch.autograd.grad([y2, ty2], x, [torch.ones_like(y)] * 2))
    # a transform around the jvp is refused, as before; a level of forward_ad without one goes the general way to the same values
    inner = lambda q: torch.func.jvp(lambda q_: sdpa_jvp(q_, x[1].detach(), x[2].detach()), (q,), (x[3].detach(),))[1].float().sum()
    with pytest.raises(RuntimeError):
        torch.func.grad(inner)(x[0].detach())
    with torch.autograd.forward_ad.dual_level():
        d = sdpa_jvp(*(torch.autograd.forward_ad.make_dual(p, t) for p, t in zip(x[:3], x[3:])))
        _equal([y, ty], list(torch.autograd.forward_ad.unpack_dual(d)))
    with pytest.raises(RuntimeError):
        torch.func.vmap(sdpa_jvp)(*(t.detach()[None] for t in x[:3]))
    with torch.no_grad():
        traced = torch.jit.trace(lambda *a: sdpa_jvp(*a), tuple(t.detach() for t in x[:3]), check_trace=False)
        assert torch.equal(traced(*(t.detach() for t in x[:3])), sdpa_jvp(*x[:3]))


def test_errors_are_those_of_the_library():
    x = [t.detach() for t in _leaves(D=48)]
    half = [t.half().requires_grad_(True) for t in x]
    with torch.no_grad():
        y = sdpa_jvp(*half[:3])
    leaf = sdpa_jvp(*half[:3])
    prev = set_kernel_family(ops.KERNELS_TCGEN05)
    try:
        for call in (lambda: sdpa_jvp(*half[:3]), lambda: torch.func.jvp(sdpa_jvp, tuple(half[:3]), tuple(t.half() for t in x[3:])),
                     lambda: torch.autograd.grad(leaf, half[:3], torch.ones_like(y))):
            with pytest.raises(_lib.JvpAttnError) as e:
                call()
            assert e.value.code == -1
    finally:
        set_kernel_family(prev)
    with pytest.raises(ValueError, match="K shape mismatch"):
        sdpa_jvp(half[0], half[1][:1], half[2])
    with pytest.raises(TypeError):
        sdpa_jvp(*(t.float() for t in x[:3]))


@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 24), (257, 40), (513, 264), (4096, 768), (16385, 3072), (2049, 2368), (100, 4608)])
def test_bias_gradient(rows, cols):
    """The sum over rows, also of a matrix with a row pitch of its own, against fp64: one rounding (2^-8) and the order of an fp32
    sum (2^-24 of the sum of magnitudes per level of adding; under 2^7 of them).  What is no plain bf16 value is summed by torch."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, b = r(rows, 16).requires_grad_(True), r(cols, 16).requires_grad_(True), r(cols).requires_grad_(True)
    plain = torch.nn.functional.linear
    for gy in (r(rows, cols), r(rows, cols + 8)[:, :cols], r(rows, cols + 1)[:, 1:], r(cols, rows).t()):
        y = dual_ops.linear(x, w, b)
        assert torch.equal(y, plain(x, w, b))
        got, want = torch.autograd.grad(y, [x, w, b], gy), torch.autograd.grad(plain(x, w, b), [x, w, b], gy)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and got[1].stride() == want[1].stride()
        ref, size = gy.double().sum(0), gy.double().abs().sum(0)
        assert bool(((got[2].double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -17 * size).all())
    gy = r(rows, cols).requires_grad_(True)

    def twice(linear):  # recorded cotangents: the second derivatives are torch's own
        once = torch.autograd.grad(linear(x, w, b), [x, w, b], gy, create_graph=True)
        return torch.autograd.grad([t.float().pow(2).sum() for t in once], [x, w, gy])

    for a, c in zip(twice(dual_ops.linear), twice(plain)):
        assert torch.equal(a, c)
    batched, = torch.autograd.grad(dual_ops.linear(x, w, b), [b], r(2, rows, cols), is_grads_batched=True)
    assert batched.shape == (2, cols)


@pytest.mark.parametrize("form", ["detached", "plain", "recorded"])
def test_inside_a_jvp_without_a_tangent(form):
    """Under a transform whose tangents do not reach the op: its value and its gradients are those of a call outside."""
    B, S, H, C = 2, 5, 4, 256
    norm = torch.nn.LayerNorm(C, device="cuda")
    lin = torch.nn.Linear(C, 24, device="cuda").bfloat16()
    cos, sin = _rand(1, S, 32, dtype=torch.float32), _rand(2, S, 32, dtype=torch.float32)
    heads = [_rand(10 + i, B, S, H, 64) for i in range(3)]
    rows = [_rand(20 + i, B, S, C) for i in range(2)]
    mods = [_rand(30 + i, B, C) for i in range(3)]
    for args, op in ((heads, safe_sdpa_jvp), ([t.transpose(1, 2) for t in heads], sdpa_jvp),
                     (rows[:1] + mods[:2], lambda x, sh, sc: dual_ops.ln_modulate(x, norm, sh, sc)), (rows + mods[:1], dual_ops.gated_residual),
                     (rows[:1], dual_ops.gelu_tanh), (rows[:1], lambda x: dual_ops.linear(x, lin.weight, lin.bias)),
                     ([_rand(40, B, S, 3, H, 64)], lambda x: torch.stack(rotary.rotary_qkv(x, cos, sin)))):
        args = [t.detach().requires_grad_(form == "recorded") for t in args]
        one = torch.ones((), device="cuda")
        inside = lambda a, *x: (op(*(t.detach() for t in x)) if form == "detached" else op(*args)) * 1.0 + 0.0 * a
        x = tuple(t.detach() for t in args)
        y, _ = torch.func.jvp(inside, (one, *x), (one, *x))
        want = op(*args)
        assert torch.equal(y.detach(), want.detach())
        if form == "recorded":
            g = _rand(50, *want.shape, dtype=want.dtype)
            _equal(torch.autograd.grad(y, args, g.to(y.dtype)), torch.autograd.grad(want, args, g))


def _jvp_or_refusal(f, prim, tang):
    try:
        return [t.detach() for t in torch.func.jvp(f, prim, tang)]
    except NotImplementedError:
        return None


@pytest.mark.parametrize("with_x", [False, True])
@pytest.mark.parametrize("which", [("weight",), ("bias",), ("weight", "bias")])
@pytest.mark.parametrize("grad", [False, True])
def test_tangents_of_parameters(which, with_x, grad):
    """A tangent on a weight or a bias either is in the result or the call is refused: never left out."""
    C = 256
    x, tx, shift, scale = (_rand(i, 2, 3, C, dtype=torch.float32) for i in range(4))
    x.requires_grad_(grad)
    for make, call, plain in (
            (lambda: torch.nn.Linear(C, 24), lambda m, a: dual_ops.linear(a, m.weight, m.bias), lambda m, a: m(a)),
            (lambda: torch.nn.LayerNorm(C), lambda m, a: dual_ops.ln_modulate(a, m, shift[:, 0], scale[:, 0]),
             lambda m, a: m(a) * (1 + scale[:, :1]) + shift[:, :1])):
        class Layer(torch.nn.Module):
            def __init__(self):
                super().__init__()
                self.inner, self.call = make().cuda(), call

            def forward(self, a):
                return self.call(self.inner, a)

        layer = Layer()
        p = dict(layer.named_parameters())
        names = [f"inner.{n}" for n in which]
        prim = tuple(p[n].detach() for n in names) + ((x,) if with_x else ())
        tang = tuple(_rand(20 + i, *t.shape, dtype=torch.float32) for i, t in enumerate(prim[:len(names)])) + ((tx,) if with_x else ())
        f = lambda *a: torch.func.functional_call(layer, dict(zip(names, a)), (a[-1] if with_x else x,))
        got = _jvp_or_refusal(f, prim, tang)
        layer.call = plain
        want = torch.func.jvp(f, prim, tang)
        if got is not None:
            assert float((got[1] - want[1]).norm()) <= 1e-5 * float(want[1].norm())


def test_tangents_of_another_kind():
    """A tangent in another type or on another device than its primal: the attention refuses it, a linear layer casts it, the rotary
    embedding goes through the operation per tensor."""
    x = [t.detach() for t in _leaves()]
    for entry in (sdpa_jvp, safe_sdpa_jvp):
        for i in range(3):
            for other, error in ((x[3 + i].float(), TypeError), (x[3 + i].half(), TypeError), (x[3 + i].cpu(), ValueError)):
                with pytest.raises(error):
                    torch.func.jvp(entry, tuple(x[:3]), tuple(other if j == i else x[3 + j] for j in range(3)))
    for grad in (False, True):
        h, w, b = (t.requires_grad_(grad) for t in (_rand(0, 2, 5, 32), _rand(1, 24, 32), _rand(2, 24)))
        th = _rand(3, 2, 5, 32, dtype=torch.float32)
        layer = lambda a: dual_ops.linear(a, w, b)
        _equal([t.detach() for t in torch.func.jvp(layer, (h,), (th,))], [t.detach() for t in torch.func.jvp(layer, (h,), (th.bfloat16(),))])
        with pytest.raises(RuntimeError):
            torch.func.jvp(layer, (h,), (th.bfloat16().cpu(),))
    qkv, tqkv, (cos, sin) = _rand(5, 2, 6, 3, 4, 64), _rand(6, 2, 6, 3, 4, 64, dtype=torch.float32), (_rand(7 + i, 6, 32, dtype=torch.float32) for i in range(2))
    q, k, v = zip(*torch.func.jvp(lambda t: rotary.rotary_qkv(t, cos, sin), (qkv,), (tqkv,)))
    for got, i in ((q, 0), (k, 1)):
        _equal(got, [rotary.apply_rotary_cast(t[:, :, i], cos, sin) for t in (qkv, tqkv)])
    _equal([t.contiguous() for t in v], [t[:, :, 2].contiguous() for t in (qkv, tqkv)])  # (Tensor.to leaves what has the type already)


def test_a_bias_alone_keeps_no_input():
    """Where only the bias wants a gradient nothing of the input or the weight is needed again, and either may be written to."""
    x, w, b = _rand(0, 4, 32), _rand(1, 24, 32), _rand(2, 24).requires_grad_(True)
    y = dual_ops.linear(x, w, b)
    x.zero_(), w.zero_()
    (db,) = torch.autograd.grad(y, [b], torch.ones_like(y))
    assert torch.equal(db, torch.full_like(db, 4.0))
    x = _rand(0, 4, 32).requires_grad_(True)
    w = _rand(1, 24, 32)
    y = dual_ops.linear(x * 1.0, w, b)
    dx, db = torch.autograd.grad(y, [x, b], torch.ones_like(y))
    assert torch.equal(dx, torch.ones_like(y) @ w) and torch.equal(db, torch.full_like(db, 4.0))


@pytest.mark.parametrize("rows,cols,launches", [(1, 768, 0), (2, 768, 2), (4096, 8, 0), (4096, 16, 2)])
def test_bias_gradient_by_torch_where_that_is_faster(rows, cols, launches):
    x, w, b = _rand(0, rows, 16), _rand(1, cols, 16), _rand(2, cols).requires_grad_(True)
    y, g = dual_ops.linear(x, w, b), _rand(3, rows, cols)
    before = _lib.launch_count()
    (db,) = torch.autograd.grad(y, [b], g)
    assert _lib.launch_count() - before == launches
    ref, size = g.double().sum(0), g.double().abs().sum(0)  # (bound as in test_bias_gradient)
    assert bool(((db.double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -17 * size).all())
