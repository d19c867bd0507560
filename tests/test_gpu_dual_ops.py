"""GPU parity of the fused (primal, tangent) pointwise ops (``semicat_b200.dual_ops``) against the PyTorch expressions they
replace (semicat/net/duo.py:128-135, 157-160), evaluated in fp32 under ``torch.func.jvp`` and differentiated in reverse
mode with cotangents on both the primal and the tangent output."""
import types

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from semicat_b200 import _lib, dual_ops


def _manual_ln(x, w, b, eps):
    mu = x.mean(-1, keepdim=True)
    xc = x - mu
    return xc * ((xc * xc).mean(-1, keepdim=True) + eps).rsqrt() * w + b


def _run(fn, primals, tangents, cots):
    leaves = [p.detach().clone().requires_grad_(True) for p in primals]
    tleaves = [None if t is None else t.detach().clone().requires_grad_(True) for t in tangents]
    idx = [i for i, t in enumerate(tleaves) if t is not None]

    def call(*dual):
        args = list(leaves)
        for i, d in zip(idx, dual):
            args[i] = d
        return fn(*args)

    y, ty = torch.func.jvp(call, tuple(leaves[i] for i in idx), tuple(tleaves[i] for i in idx))
    wrt = leaves + [t for t in tleaves if t is not None]
    grads = torch.autograd.grad([y, ty], wrt, [cots[0].to(y.dtype), cots[1].to(ty.dtype)], allow_unused=True)
    return y, ty, grads


def _close(a, b, what, rtol, atol):
    if a is None or b is None:
        assert a is None and b is None or (b is None and float(a.abs().max()) == 0) or (a is None and float(b.abs().max()) == 0), what
        return
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    assert bool((err <= tol).all()), f"{what}: max err {err.max().item():.3e} (ref max {b.abs().max().item():.3e})"


def _ln_inputs(B, S, C, dtype, seed=0, tx=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, t = r(B, S, C).to(dtype), (r(B, S, C).to(dtype) if tx else None)
    mod = (r(B, 1, 6 * C) * 0.5).to(dtype)  # chunks of one projection, as in the denoiser: strided (B, 1, C) views
    tmod = (r(B, 1, 6 * C) * 0.5).to(dtype)
    sh, sc = mod[..., :C], mod[..., C:2 * C]
    tsh, tsc = tmod[..., :C], tmod[..., C:2 * C]
    norm = torch.nn.LayerNorm(C).cuda()
    with torch.no_grad():
        norm.weight.copy_(1.0 + 0.3 * r(C))
        norm.bias.copy_(0.2 * r(C))
    cots = (r(B, S, C), r(B, S, C))
    return x, t, sh, sc, tsh, tsc, norm, cots


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("shape", [(3, 40, 768), (2, 17, 256), (1, 128, 1024)])
def test_ln_modulate_fp32_matches_pytorch(shape, exact):
    B, S, C = shape
    x, t, sh, sc, tsh, tsc, norm, cots = _ln_inputs(B, S, C, torch.float32)
    w, b = norm.weight, norm.bias
    if exact:
        ref_fn = lambda x_, sh_, sc_, w_, b_: _manual_ln(x_, w_, b_, norm.eps) * (1.0 + sc_) + sh_
    else:  # PyTorch's own LayerNorm: its forward-mode formula holds mean / rstd constant when differentiated again
        ref_fn = lambda x_, sh_, sc_, w_, b_: F.layer_norm(x_, (C,), w_, b_, norm.eps) * (1.0 + sc_) + sh_

    def fused(x_, sh_, sc_, w_, b_):
        # the public entry point with the LayerNorm weight and bias as differentiable leaves
        stand_in = types.SimpleNamespace(weight=w_, bias=b_, eps=norm.eps, normalized_shape=(C,))
        return dual_ops.ln_modulate(x_, stand_in, sh_, sc_, exact=exact)

    before = _lib.launch_count()
    got = _run(fused, (x, sh, sc, w, b), (t, tsh, tsc, None, None), cots)
    # primal and tangent forward; one backward kernel per cotangent (the second adds to dx); one launch for the
    # gradients of the modulation tensors and the LayerNorm parameters
    assert _lib.launch_count() - before == 5
    want = _run(ref_fn, (x, sh, sc, w, b), (t, tsh, tsc, None, None), cots)
    _close(got[0], want[0], "y", 1e-4, 1e-4)
    _close(got[1], want[1], "ty", 1e-4, 1e-4)
    for name, a, r in zip(("dx", "dshift", "dscale", "dgamma", "dbeta", "dtx", "dtshift", "dtscale"), got[2], want[2]):
        _close(a, r, f"{name} (exact={exact})", 2e-3, 2e-3 * float(r.abs().max()))


def test_ln_modulate_bf16_and_missing_tangent_on_x():
    """bf16 tensors as under autocast; the first block of the denoiser sees a tangent on the modulation only."""
    B, S, C = 4, 64, 768
    for tx in (True, False):
        x, t, sh, sc, tsh, tsc, norm, cots = _ln_inputs(B, S, C, torch.bfloat16, seed=3, tx=tx)
        fused = lambda x_, sh_, sc_: dual_ops.ln_modulate(x_, norm, sh_, sc_)
        ref_fn = lambda x_, sh_, sc_: F.layer_norm(x_.float(), (C,), norm.weight, norm.bias, norm.eps) * (1.0 + sc_.float()) + sh_.float()
        got = _run(fused, (x, sh, sc), (t, tsh, tsc), cots)
        want = _run(ref_fn, (x, sh, sc), (t, tsh, tsc), cots)
        assert got[0].dtype == torch.bfloat16
        _close(got[0], want[0], "y", 2e-2, 2e-2)
        _close(got[1], want[1], "ty", 2e-2, 4e-2)
        for name, a, r in zip(("dx", "dshift", "dscale", "dtx", "dtshift", "dtscale") if tx else ("dx", "dshift", "dscale", "dtshift", "dtscale"),
                              got[2], want[2]):
            _close(a, r, f"{name} (tx={tx})", 3e-2, 3e-2 * float(r.float().abs().max()))


@pytest.mark.parametrize("cotangents", ["both", "tangent", "primal"])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("tx", [True, False])
def test_ln_modulate_bf16_launches_and_gradients(tx, exact, cotangents):
    """The bf16 pair through the public entry point: one kernel forward, one for whichever cotangents arrive, one finalize, and
    every gradient against fp64.  bf16 results to one rounding (2^-8; 2^-7 where values that were rounded themselves
    enter), fp32 parameter gradients to the order of their sums."""
    B, S, C = 3, 50, 768
    x, t, sh, sc, tsh, tsc, norm, cots = _ln_inputs(B, S, C, torch.bfloat16, seed=11, tx=tx)
    cots = [c.to(torch.bfloat16) for c in cots]
    names = ["x", "shift", "scale"] + ["tx"] * tx + ["tshift", "tscale", "gamma", "beta"]

    def run(leaf, layer_norm):
        prim = [leaf(v) for v in (x, sh, sc)]
        tang = [leaf(v) for v in (t, tsh, tsc) if v is not None]
        w, b = (v.detach().clone().to(torch.float32 if leaf is same else torch.float64).requires_grad_(True) for v in (norm.weight, norm.bias))
        duals, rest = (prim, []) if tx else (prim[1:], prim[:1])
        y, ty = torch.func.jvp(lambda *d: layer_norm(*rest, *d, w, b), tuple(duals), tuple(tang))
        outs, gs = {"both": ([y, ty], cots), "tangent": ([ty], cots[1:]), "primal": ([y], cots[:1])}[cotangents]
        grads = torch.autograd.grad(outs, [*prim, *tang, w, b], [g.to(y.dtype) for g in gs], allow_unused=True)
        return y, ty, dict(zip(names, grads))

    same = lambda v: v.detach().clone().requires_grad_(True)
    double = lambda v: v.detach().double().requires_grad_(True)
    ours = lambda x_, sh_, sc_, w, b: dual_ops.ln_modulate(
        x_, types.SimpleNamespace(weight=w, bias=b, eps=norm.eps, normalized_shape=(C,)), sh_, sc_, exact=exact)
    ref_ln = (lambda v, w, b: _manual_ln(v, w, b, norm.eps)) if exact else (lambda v, w, b: F.layer_norm(v, (C,), w, b, norm.eps))
    before = _lib.launch_count()
    y, ty, got = run(same, ours)
    assert _lib.launch_count() - before == 3
    y_ref, ty_ref, want = run(double, lambda x_, sh_, sc_, w, b: ref_ln(x_, w, b) * (1 + sc_) + sh_)
    _close(y, y_ref, "y", 2 ** -8, 1e-4)
    _close(ty, ty_ref, "ty", 2 ** -8, 1e-4)
    for n in names:
        if want[n] is None:
            assert got[n] is None or not got[n].any(), n
            continue
        peak = float(want[n].abs().max())
        _close(got[n], want[n], f"{n} (tx={tx}, exact={exact}, {cotangents})", 2 ** -7 if n not in ("gamma", "beta") else 1e-5, 1e-4 * peak)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_residual_matches_pytorch(dtype):
    B, S, C = 3, 50, 768
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)
    x, y, tx, ty = r(B, S, C), r(B, S, C), r(B, S, C), r(B, S, C)
    gates, tgates = r(B, 1, 6 * C), r(B, 1, 6 * C)
    gate, tgate = gates[..., 2 * C:3 * C], tgates[..., 2 * C:3 * C]
    cots = (torch.randn(B, S, C, device="cuda", generator=g), torch.randn(B, S, C, device="cuda", generator=g))
    fused = lambda x_, y_, g_: dual_ops.gated_residual(x_, y_, g_, p=0.1, training=False)
    ref_fn = lambda x_, y_, g_: y_.float() * g_.float() + x_.float()
    before = _lib.launch_count()
    got = _run(fused, (x, y, gate), (tx, ty, tgate), cots)
    assert _lib.launch_count() - before == 2  # one kernel for (z, tz), one for both cotangents
    want = _run(ref_fn, (x, y, gate), (tx, ty, tgate), cots)
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    _close(got[0], want[0], "z", tol, tol)
    _close(got[1], want[1], "tz", tol, 2 * tol)
    for name, a, rr in zip(("dx", "dy", "dgate", "dtx", "dty", "dtgate"), got[2], want[2]):
        _close(a, rr, name, tol, tol * float(rr.float().abs().max()) + 1e-6)


def test_gated_residual_dropout_uses_one_mask_for_primal_and_tangent():
    B, S, C = 2, 64, 512
    g = torch.Generator(device="cuda").manual_seed(9)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, y, tx, ty, gate = r(B, S, C), r(B, S, C), r(B, S, C), r(B, S, C), r(B, 1, C)
    z, tz = torch.func.jvp(lambda x_, y_: dual_ops.gated_residual(x_, y_, gate, p=0.25, training=True), (x, y), (tx, ty))
    kept = (z - x) != 0
    frac = kept.float().mean().item()
    assert 0.70 < frac < 0.80, frac
    assert torch.allclose((z - x)[kept], (y * gate / 0.75)[kept], rtol=1e-5, atol=1e-6)
    assert torch.equal((tz - tx) != 0, kept)  # same mask
    assert torch.allclose((tz - tx)[kept], (ty * gate / 0.75)[kept], rtol=1e-5, atol=1e-6)


def test_unsupported_shapes_fall_back_to_pytorch():
    x = torch.randn(2, 8, 96, device="cuda")
    norm = torch.nn.LayerNorm(96).cuda()
    sh, sc = torch.randn(2, 1, 96, device="cuda"), torch.randn(2, 1, 96, device="cuda")
    before = _lib.launch_count()
    y = dual_ops.ln_modulate(x, norm, sh, sc)
    assert _lib.launch_count() == before
    assert torch.allclose(y, norm(x) * (1 + sc) + sh)
    z = dual_ops.gated_residual(x, x, sc)
    assert torch.allclose(z, x * sc + x)


@pytest.mark.parametrize("dtype,V,pad", [(torch.float32, 27, 0), (torch.bfloat16, 30522, 6), (torch.float32, 1000, 0)])
def test_flow_map_head_matches_pytorch(dtype, V, pad):
    """xst = x + dt (softmax(l) - x) and its derivative in t, with cotangents on both, against the PyTorch expression in
    fp32; the 30522-wide case reads the logits as a view of a padded (…, 30528) projection output, as the denoiser does."""
    B, L = 3, 5
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    lfull, tlfull = (2.0 * r(B, L, V + pad)).to(dtype), r(B, L, V + pad).to(dtype)
    l, tl = lfull[..., :V], tlfull[..., :V]
    x = r(B, L, V)
    t = torch.rand(B, device="cuda", generator=g) * 0.8 + 0.1
    s = torch.rand(B, device="cuda", generator=g) * t
    cots = (r(B, L, V), r(B, L, V))

    def run(fn):
        ll, tll = l.detach().clone().requires_grad_(True), tl.detach().clone().requires_grad_(True)
        tt = t.clone()

        def f(l_, t_):
            dt = (t_ - s) / (1.0 - s + 1e-8)
            return fn(l_, x, dt)

        xst, dv = torch.func.jvp(f, (ll, tt), (tll, torch.ones_like(tt)))
        grads = torch.autograd.grad([xst, dv], [ll, tll], list(cots))
        return xst, dv, grads

    before = _lib.launch_count()
    got = run(dual_ops.flow_map_head)
    assert _lib.launch_count() - before == 4
    want = run(lambda l_, x_, dt: x_ + dt.view(-1, 1, 1) * (l_.float().softmax(dim=-1) - x_))
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    _close(got[0], want[0], "xst", tol, 1e-5)
    _close(got[1], want[1], "dv", tol, 1e-4 if dtype == torch.float32 else 1e-3)
    for name, a, b in zip(("dlogits", "dtlogits"), got[2], want[2]):
        _close(a, b, name, tol, (1e-5 if dtype == torch.float32 else 2e-2) * float(b.float().abs().max()))


def test_generated_dropout_masks_are_consistent_between_passes_and_have_the_right_rate():
    """Inside ``dropout_seed`` the kernels regenerate each call's keep mask from (seed, call number): forward, tangent and
    backward of one call must see the same mask, different calls and different steps different ones."""
    B, S, C, p = 4, 64, 768, 0.25
    dev = "cuda"
    x = torch.zeros(B, S, C, device=dev)
    ones = torch.ones(B, S, C, device=dev)
    gate = torch.ones(B, 1, C, device=dev)
    masks = []
    for _ in range(2):  # two "steps"
        with dual_ops.dropout_seed(torch.device(dev)):
            # call 0: primal-only path; z = mask, and d z / d y = mask
            y = ones.clone().requires_grad_(True)
            z = dual_ops.gated_residual(x, y, gate, p, True)
            (gy,) = torch.autograd.grad(z, y, ones)
            assert torch.equal(z.detach(), gy)
            # call 1: (primal, tangent) path with tangent 1 on the branch only: z = tz = mask, gradients = mask
            y2, t2 = ones.clone().requires_grad_(True), ones.clone().requires_grad_(True)
            z2, tz2 = torch.func.jvp(lambda y_: dual_ops.gated_residual(x, y_, gate, p, True), (y2,), (t2,))
            assert torch.equal(z2.detach(), tz2.detach())
            g_y2, g_t2 = torch.autograd.grad([z2, tz2], [y2, t2], [ones, ones])
            assert torch.equal(g_y2, z2.detach()) and torch.equal(g_t2, z2.detach())
            masks += [z.detach(), z2.detach()]
    for m in masks:
        kept = m != 0
        assert torch.allclose(m[kept], torch.full_like(m[kept], 1.0 / (1.0 - p)))
        assert abs(float((~kept).float().mean()) - p) < 0.01  # 196608 draws: sigma = 0.001
    for i in range(4):
        for j in range(i + 1, 4):
            assert not torch.equal(masks[i], masks[j])
    assert _lib.device_status() == 0


@pytest.mark.parametrize("shape", [(1, 1, 256), (3, 17, 512), (2, 50, 768), (5, 130, 1024), (40, 33, 768)])
@pytest.mark.parametrize("missing", ["none", "x", "scale", "shift"])
@pytest.mark.parametrize("exact", [False, True])
def test_ln_modulate_bf16_pair_kernels_match_the_single_ones(shape, missing, exact):
    """The one-pass bf16 kernels against the kernels that take primal and tangent one at a time: y, ty and dtx are rounded
    once in either form (so at most neighbouring bf16 values, 2^-7 relative), dx twice by the single kernels (2^-7 of its two
    parts), the fp32 column sums differ in their order only."""
    B, S, C = shape
    x, t, sh, sc, tsh, tsc, norm, cots = _ln_inputs(B, S, C, torch.bfloat16, seed=C + S, tx=missing != "x")
    tsh, tsc = None if missing == "shift" else tsh, None if missing == "scale" else tsc
    w, b = norm.weight.detach().float(), norm.bias.detach().float()
    g, gt = (c.to(torch.bfloat16) for c in cots)
    new = lambda: torch.full_like(x, float("nan"))
    stat = lambda: torch.full((B * S,), float("nan"), device="cuda")
    y, ty, mean, rstd = new(), new(), stat(), stat()
    dual_ops._ln_dual_launch(0, x, t, w, b, sh, sc, tsh, tsc, mean, rstd, y, ty, None, None, None, None, None, norm.eps, exact)
    y1, ty1, mean1, rstd1 = new(), new(), stat(), stat()
    tz = torch.zeros_like(x) if t is None else t
    dual_ops._ln_launch(0, x, None, w, b, sh, sc, None, None, mean1, rstd1, y1, None, None, None, None, norm.eps, exact)
    dual_ops._ln_launch(1, x, tz, w, b, None, sc, tsh, tsc, mean1, rstd1, ty1, None, None, None, None, norm.eps, exact)
    _close(mean, mean1, "mean", 1e-5, 1e-6)
    _close(rstd, rstd1, "rstd", 1e-5, 1e-6)
    _close(y, y1, "y", 2 ** -7, 1e-5)
    _close(ty, ty1, "ty", 2 ** -7, 1e-4)
    sums, sums1 = (torch.zeros(5, B, C, device="cuda") for _ in range(2))
    dx, dtx, dx1, dtx1 = new(), new(), new(), new()
    dual_ops._ln_dual_launch(1, x, t, w, None, None, sc, None, tsc, mean, rstd, None, None, g, gt, dx, dtx, sums, norm.eps, exact)
    dual_ops._ln_launch(2, x, None, w, None, None, sc, None, None, mean, rstd, None, g, dx1, None, sums1[:2], norm.eps, exact)
    first = dx1.float().abs()
    dual_ops._ln_launch(3, x, tz, w, None, None, sc, None, tsc, mean, rstd, None, gt, dx1, dtx1, sums1[2:], norm.eps, int(exact) | 2)
    _close(dtx, dtx1, "dtx", 2 ** -7, 1e-4)
    err = (dx.float() - dx1.float()).abs()
    assert bool((err <= 2 ** -7 * (first + dx1.float().abs()) + 1e-4).all()), err.max()
    sums1[0] += sums1[4]  # the pair kernel keeps sum(g n) + sum(gt nd) together
    scale = sums1[:4].abs().max()
    assert float((sums[:4] - sums1[:4]).abs().max()) <= 1e-5 * float(scale) * S ** 0.5 and not sums[4].any()


@pytest.mark.parametrize("shape", [(600, 9, 768), (128, 50, 256), (37, 130, 1024), (1500, 4, 512), (1500, 3, 512)])
@pytest.mark.parametrize("missing", ["none", "x", "scale", "shift"])
def test_ln_modulate_bf16_pair_kernels_with_rows_walked(shape, missing):
    """The same where a warp walks several rows of a sample, some fewer than others, and on both sides of the fewest rows for that."""
    test_ln_modulate_bf16_pair_kernels_match_the_single_ones(shape, missing, False)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 1, 256), (1100, 3, 768), (9, 50, 512), (2, 128, 1024), (600, 8, 768), (1200, 9, 256),
                                   (300, 50, 1024), (75, 128, 768), (148, 129, 512)])
def test_primal_ln_and_gate_over_the_ways_rows_are_split(shape, dtype):
    """Without tangents a row per warp or several, a few rows per CTA or many, by the number of samples and rows: results and
    gradients against fp64.  bf16 results to one rounding (2^-8), fp32 ones and the column sums to the order of the sums."""
    B, S, C = shape
    x, y, sh, ga, _, _, norm, (gh, gz) = _ln_inputs(B, S, C, dtype, seed=B + S)
    sc = ga * 0.5
    gh, gz = gh.to(dtype), gz.to(dtype)
    leaves = [v.detach().clone().requires_grad_(True) for v in (x, y, sh, sc, ga)]
    w, b = norm.weight, norm.bias
    h = dual_ops.ln_modulate(leaves[0], norm, leaves[2], leaves[3])
    z = dual_ops.gated_residual(leaves[0], leaves[1], leaves[4], p=0.0, training=True)
    got = torch.autograd.grad([h, z], [*leaves[1:], w, b], [gh, gz], retain_graph=True)
    dx_h, = torch.autograd.grad(h, leaves[0], gh)
    ref = [v.detach().double().requires_grad_(True) for v in (x, y, sh, sc, ga, w, b)]
    hr = F.layer_norm(ref[0], (C,), ref[5], ref[6], norm.eps) * (1 + ref[3]) + ref[2]
    zr = ref[0] + ref[4] * ref[1]
    want = torch.autograd.grad([hr, zr], ref[1:], [gh.double(), gz.double()], retain_graph=True)
    dxr_h, = torch.autograd.grad(hr, ref[0], gh.double())
    tol = 2 ** -8 if dtype == torch.bfloat16 else 1e-5
    _close(h, hr, "h", tol, 1e-4 if dtype == torch.bfloat16 else 1e-5)
    _close(z, zr, "z", tol, 1e-5)
    _close(dx_h, dxr_h, "dx", tol, 1e-4 * float(dxr_h.abs().max()))
    for n, a, r in zip(("dy", "dshift", "dscale", "dgate", "dgamma", "dbeta"), got, want):
        _close(a, r, n, tol if n not in ("dgamma", "dbeta") else 1e-5, 1e-4 * float(r.abs().max()))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("dtype,other", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float16)])
@pytest.mark.parametrize("grad", [False, True])
def test_tangents_of_another_type(dtype, other, grad):
    """A tangent in another type than its primal counts as that value in the primal's type; one on another device is refused."""
    g = torch.Generator(device="cuda").manual_seed(0)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g)
    B, S, C, V = 2, 5, 256, 40
    norm = torch.nn.LayerNorm(C, device="cuda")
    dt = torch.rand(B, device="cuda", generator=g)
    data = mk(B, S, V)
    for op, shapes in ((lambda x, sh, sc: dual_ops.ln_modulate(x, norm, sh, sc), [(B, S, C), (B, 1, C), (B, 1, C)]),
                       (dual_ops.gated_residual, [(B, S, C), (B, S, C), (B, C)]), (dual_ops.gelu_tanh, [(B, S, C)]),
                       (lambda l: dual_ops.flow_map_head(l, data, dt), [(B, S, V)])):
        prim = tuple(mk(*s).to(dtype).requires_grad_(grad) for s in shapes)
        tang = tuple(mk(*s).to(other) for s in shapes)
        y, ty = torch.func.jvp(op, prim, tang)
        want = torch.func.jvp(op, prim, tuple(t.to(dtype) for t in tang))
        assert ty.dtype == want[1].dtype and torch.equal(y, want[0]) and torch.equal(ty, want[1])
        if grad:
            cots = [mk(*y.shape).to(y.dtype) for _ in range(2)]
            for a, b in zip(torch.autograd.grad([y, ty], prim, cots), torch.autograd.grad(want, prim, cots)):
                # (column sums are added by atomics in any order, and rounded once)
                assert torch.allclose(a.float(), b.float(), rtol=2 ** -7, atol=1e-5)
        for i in range(len(prim)):
            with pytest.raises((ValueError, RuntimeError)):
                torch.func.jvp(op, prim, tuple(t.to(dtype).cpu() if j == i else t.to(dtype) for j, t in enumerate(tang)))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B", [262139, 262141, 524289])
def test_ln_modulate_gradients_of_many_samples(B):
    """One row per sample: the gradient of shift is the cotangent itself, that of scale the cotangent times the normalised row
    (one rounding to 16 bits, 2^-8, and fp32 sums below it)."""
    C = 256
    g = torch.Generator(device="cuda").manual_seed(0)
    mk = lambda: torch.randn(B, 1, C, device="cuda", generator=g).bfloat16()
    norm = torch.nn.LayerNorm(C, device="cuda")
    x, gy, shift, scale = mk(), mk(), mk().requires_grad_(True), mk().requires_grad_(True)
    y = dual_ops.ln_modulate(x, norm, shift, scale)
    d_shift, d_scale = torch.autograd.grad(y, [shift, scale], gy)
    assert torch.equal(d_shift, gy)
    want = torch.nn.functional.layer_norm(x.float(), (C,)) * gy.float()
    assert bool(((d_scale.float() - want).abs() <= 2 ** -7 * want.abs() + 1e-5).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("which", ["x", "shift", "weight", "bias", "cotangent"])
def test_ln_modulate_refuses_rows_off_the_16_byte_grid(dtype, which):
    """The kernels read 16 bytes at a time: contiguous tensors that start between two such places are refused, as by the other ops."""
    B, S, C = 2, 5, 256
    off = lambda t: torch.cat((t.flatten()[:1], t.flatten()))[1:].view(t.shape)
    place = lambda name, t: off(t) if name == which else t
    norm = torch.nn.LayerNorm(C, device="cuda")
    norm.weight = torch.nn.Parameter(place("weight", torch.ones(C, device="cuda")))
    norm.bias = torch.nn.Parameter(place("bias", torch.ones(C, device="cuda")))
    x, shift, scale = place("x", torch.ones(B, S, C, device="cuda", dtype=dtype)), *(place(n, torch.ones(B, C, device="cuda", dtype=dtype)) for n in ("shift", "scale"))

    def refused(f):
        with pytest.raises(_lib.JvpAttnError) as e:
            f()
        assert e.value.code == -3

    if which == "cotangent":
        y = dual_ops.ln_modulate(x.requires_grad_(True), norm, shift, scale)
        refused(lambda: torch.autograd.grad(y, [x], off(torch.ones_like(y))))
    else:
        call = lambda a: dual_ops.ln_modulate(a, norm, shift, scale)
        with torch.no_grad():
            refused(lambda: call(x))
        refused(lambda: torch.func.jvp(call, (x,), (torch.ones_like(x),)))
        refused(lambda: call(x.detach().requires_grad_(True)))
    assert _lib.device_status() == 0
