"""16-bit copies of a model's parameters in one launch: bit for bit what ``Tensor.to`` and zero padding give, over vectors and
matrices whose sizes are no multiple of anything, and the denoiser's pass that uses them against the one that does not."""
import pytest
import torch

from semicat_b200 import _lib, _nodes, train_step, vocab_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_copies(dtype):
    g = torch.Generator(device="cuda").manual_seed(0)
    base = torch.randn(4099, device="cuda", generator=g)
    shapes = [(1,), (7,), (8,), (4608,), (1, 1), (3, 5), (9, 16), (768, 1003), (30, 30522), (33, 8200), (0,), (5, 0)] + [(17, 24)] * 60
    params = [torch.randn(s, device="cuda", generator=g) * 3 for s in shapes] + [base[3:4000], base[2:4098]]  # and off the 16-byte grid
    for align in (False, True):
        flags, scale = [align] * len(params), [1.0 + 0.37 * (i % 3) for i in range(len(params))]
        out = _nodes.module().cast_params(params, scale, flags, dtype == torch.bfloat16)
        for p, s, o in zip(params, scale, out):
            want = (p * s).to(dtype)
            pad = [(-n) % 8 if align else 0 for n in (p.shape if p.dim() == 2 else (1, *p.shape))]
            want = torch.nn.functional.pad(want, (0, pad[1], 0, pad[0]) if p.dim() == 2 else (0, pad[1]))
            assert o.shape == want.shape and o.dtype == dtype and o.data_ptr() % 16 == 0 and torch.equal(o, want)
    assert _nodes.module().cast_params([base.half()], [1.0], [False], True) is None
    assert _nodes.module().cast_params([torch.ones(4, 4, device="cuda").t()[:2]], [1.0], [False], True) is None
    assert _lib.device_status() == 0


@pytest.mark.parametrize("V,B,L,dtype", [(1003, 3, 40, torch.bfloat16), (1024, 2, 64, torch.bfloat16), (27, 2, 33, torch.bfloat16), (1003, 2, 40, torch.float16)])
@pytest.mark.parametrize("attention", ["lib", "sdpa"])
def test_pass(monkeypatch, V, B, L, dtype, attention):
    torch.manual_seed(0)
    with torch.device("cuda"):
        net = train_step.DiT(V, 256, 64, 3, 4, dropout=0.0, length=L, embed_type="rms" if V < 512 else "naive")
    train_step.randomise_zero_init(net)
    net.eval()
    x1 = torch.randint(0, V, (B, L), device="cuda")
    noise = train_step.draw_noise(x1, V)
    s, t = noise["u_sd"] * noise["t_sd"], noise["t_sd"]
    plain = train_step.interpolate(noise["x0"], x1, s.view(-1, 1, 1))
    inputs = [plain] if V < 512 or dtype == torch.float16 else [plain, vocab_ops.interpolate_cast(noise["x0"], x1, s)]
    used = []
    of, chained = train_step._PassCasts.of, train_step._PassCasts.chained
    for x in inputs:
        out = []
        for way, chain in ((lambda *a: (used.append(of(*a)), used[-1])[1], True), (of, False), (lambda *a: None, False)):
            monkeypatch.setattr(train_step._PassCasts, "of", staticmethod(way))
            if not chain:
                monkeypatch.setattr(train_step._PassCasts, "chained", staticmethod(lambda n: False))
            with torch.no_grad(), torch.autocast("cuda", dtype=dtype):
                out.append(net(x, s, t, attention=attention, padded_logits=True))
            monkeypatch.setattr(train_step._PassCasts, "chained", staticmethod(chained))
        assert float((out[0] - out[2]).float().norm() / out[2].float().norm()) < 2 ** -8
        # the modulation comes from another GEMM (16-bit results, 64 terms): half a unit of 2^-8 now and then, through three blocks
        assert out[0].shape == out[1].shape and out[0].dtype == out[1].dtype
        assert float((out[0] - out[1]).float().norm() / out[1].float().norm()) < 2 ** -8
    assert all(u is not None for u in used)
    # (the blocks as one chain, or one by one where somebody listens or drops out)
    assert chained(net)
    handle = net.blocks[1].register_forward_hook(lambda *a: None)
    assert not chained(net)
    handle.remove()
    net.blocks[0].drop.p = 0.5
    assert chained(net) and not chained(net.train())
    net.blocks[0].drop.p = 0.0
    net.eval()
    with torch.autocast("cuda", dtype=dtype):  # gradients may be wanted: not for this pass
        assert of(net, plain, attention) is None
    with torch.no_grad():
        assert of(net, plain, attention) is None
        with torch.autocast("cuda", dtype=dtype):
            assert of(net.half(), plain, attention) is None


def _small(width=256, blocks=2, V=1003, L=32, **kw):
    torch.manual_seed(0)
    with torch.device("cuda"):
        net = train_step.DiT(V, width, 64, blocks, width // 64, dropout=0.0, length=L, **kw)
    train_step.randomise_zero_init(net)
    x1 = torch.randint(0, V, (2, L), device="cuda")
    noise = train_step.draw_noise(x1, V)
    s, t = noise["u_sd"] * noise["t_sd"], noise["t_sd"]
    return net.eval(), train_step.interpolate(noise["x0"], x1, s.view(-1, 1, 1)), s, t


def _pass(net, x, s, t, **kw):
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        return net(x, s, t, attention="lib", **kw)


@pytest.mark.parametrize("width", [64, 128, 384])
def test_pass_of_widths_without_a_kernel(monkeypatch, width):
    """Widths that the LayerNorm and gate kernels do not take: the pass is that of autocast."""
    net, *inputs = _small(width)
    out = _pass(net, *inputs)
    monkeypatch.setattr(train_step._PassCasts, "of", staticmethod(lambda *a: None))
    want = _pass(net, *inputs)
    assert out.shape == want.shape and out.dtype == want.dtype
    assert float((out - want).float().norm() / want.float().norm()) < 2 ** -8  # as in test_pass


class _Wrapped(torch.nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, x, cos, sin, c, attention):
        return self.inner(x, cos, sin, c, attention)


class _FiveArguments(train_step.Block):
    def forward(self, x, cos, sin, c, attention):
        return super().forward(x, cos, sin, c, attention)


def _changes(net, what):
    blk = net.blocks[0]
    if what == "wrapper":
        net.blocks[0] = _Wrapped(blk)
    elif what == "subclass":
        blk.__class__ = _FiveArguments
    elif what == "pre-hook":
        blk.register_forward_pre_hook(lambda m, a: (*a[:3], a[3] * 2.0, *a[4:]))
    elif what == "hook with arguments":
        blk.register_forward_hook(lambda m, a, out: out * float(len(a)))
    elif what == "own forward":
        blk.forward = lambda x, cos, sin, c, attention: x
    elif what == "ada without bias":
        blk.ada.bias = None
    elif what == "head without bias":
        net.head.bias = None
    elif what == "embedding hook":
        net.embed.register_forward_pre_hook(lambda m, a: tuple(a) if len(a) == 3 else 1 / 0)
    elif what == "embedding subclass":
        class Embed(train_step.NaiveEmbed):
            def forward(self, x, t, cond):
                return super().forward(x, t, cond)
        net.embed.__class__ = Embed
    elif what == "norm without weight":
        blk.norm1 = torch.nn.LayerNorm(256, elementwise_affine=False)
    elif what == "norm in bf16":
        blk.norm2.bfloat16()
    elif what == "no blocks":
        net.blocks = torch.nn.ModuleList()


@pytest.mark.parametrize("what", ["wrapper", "subclass", "pre-hook", "hook with arguments", "own forward", "ada without bias", "head without bias",
                                  "embedding hook", "embedding subclass", "norm without weight", "norm in bf16", "no blocks"])
def test_pass_of_changed_models(monkeypatch, what):
    """What a program has made of the model's parts is what runs."""
    net, *inputs = _small()
    plain = _pass(net, *inputs)
    _changes(net, what)
    out = _pass(net, *inputs)
    monkeypatch.setattr(train_step._PassCasts, "of", staticmethod(lambda *a: None))
    want = _pass(net, *inputs)
    assert float((out - want).float().norm() / want.float().norm()) < 2 ** -8  # as in test_pass
    if what in ("pre-hook", "hook with arguments", "own forward", "no blocks"):
        assert float((plain - want).float().norm() / want.float().norm()) > 2 ** -5


def test_modes_see_the_copies():
    """Under a dispatch mode the pass makes its copies with torch's own operations, which the mode sees."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Casts(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen += "_to_copy" in str(func)
            return func(*args, **(kwargs or {}))

    net, *inputs = _small()
    with torch.no_grad():
        want = [m.weight.bfloat16() for m in net.modules() if isinstance(m, torch.nn.Linear)]
        with Casts() as mode:
            assert _nodes.module().cast_params([net.head.weight], [1.0], [False], True) is None
            _pass(net, *inputs)
    assert mode.seen >= len(want)
