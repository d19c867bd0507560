"""Backward over many (batch, head) items per CTA with a single tile of keys: each item's rows and row statistics must
stay in place until every warp has read them, however little work an item has."""
import pytest
import torch

import gpu_util as G
from semicat_b200 import _lib, ops

pytestmark = pytest.mark.gpu

B, H, LQ = 5, 128, 128  # 640 items of 128 rows: at least four per CTA on 148 SMs


def _backward(ins, mode):
    t = {n: G.place(ins[n], torch.bfloat16, "bshd") for n in G.IN_NAMES}
    g_o = G.place(ins["g_o"], torch.bfloat16, "bshd") if mode in ("both", "pri") else None
    g_to = G.place(ins["g_od"], torch.bfloat16, "bshd") if mode in ("both", "tan") else None
    o, to = torch.empty_like(t["q"]), torch.empty_like(t["q"])
    b, h = t["q"].shape[:2]
    lse = torch.zeros(b, h, ops.stat_len(LQ), device="cuda")
    mu = torch.zeros_like(lse)
    ops.jvp_attention_fwd(*[t[n] for n in G.IN_NAMES], o, to, lse, mu)
    grads = [torch.full_like(t[n], G.CANARY) for n in G.IN_NAMES]
    if mode == "pri":
        ops.jvp_attention_bwd(t["q"], t["k"], t["v"], None, None, None, o, None, g_o, None, lse, None, *grads[:3])
        return dict(zip(G.GRAD_NAMES, grads[:3]))
    ops.jvp_attention_bwd(*[t[n] for n in G.IN_NAMES], o, to, g_o, g_to, lse, mu, *grads)
    return dict(zip(G.GRAD_NAMES, grads))


@pytest.mark.parametrize("mode", ["both", "tan", "pri"])
@pytest.mark.parametrize("Lk", [1, 33, 64])
@pytest.mark.parametrize("D", [64, 72, 96, 128])
def test_many_items_with_one_key_tile(D, Lk, mode):
    """Against the same heads one item per CTA (128 items; an item's arithmetic does not depend on its place, so bit for
    bit) and, for sampled heads, the oracle."""
    ins = G.rounded(G.synth(B, H, LQ, Lk, D, seed=D + Lk), torch.bfloat16)
    got = _backward(ins, mode)
    for b in range(B):
        alone = _backward({n: x[b:b + 1] for n, x in ins.items()}, mode)
        for n in alone:
            assert torch.equal(got[n][b], alone[n][0]), (n, b)
    heads = slice(3, None, 41)
    sub = {n: x[:, heads] for n, x in ins.items()}
    want = G.oracle(sub, mode)
    for n in got:
        G.assert_close(got[n][:, heads].float().cpu().numpy(), want[n], f"{n} D={D} Lk={Lk} {mode}")
    assert _lib.device_status() == 0


@pytest.mark.parametrize("tangents", [True, False])
@pytest.mark.parametrize("ntiles", [1, 2, 3, 5])
@pytest.mark.parametrize("D", [72, 128])
def test_forward_at_few_key_tiles(D, ntiles, tangents):
    """Heads wider than 64 channels alternate between two score regions; the last value products may be over before a warp
    asks for them.  Many CTAs, several times: every call complete, equal and close to the oracle on sampled heads."""
    ins = G.rounded(G.synth(B, H, LQ, 64 * ntiles - 5, D, seed=D + ntiles), torch.bfloat16)
    t = {n: G.place(ins[n], torch.bfloat16, "bshd") for n in G.IN_NAMES}
    first = None
    for _ in range(4):
        o, to = torch.full_like(t["q"], G.CANARY), torch.full_like(t["q"], G.CANARY) if tangents else None
        lse = torch.full((B, H, ops.stat_len(LQ)), G.CANARY, device="cuda")
        mu = torch.full_like(lse, G.CANARY) if tangents else None
        tang = [t[n] if tangents else None for n in ("tq", "tk", "tv")]
        ops.jvp_attention_fwd(t["q"], t["k"], t["v"], *tang, o, to, lse, mu)
        out = [x for x in (o, to, lse, mu) if x is not None]
        first = first or out
        assert all(torch.equal(x, y) for x, y in zip(out, first))
    heads = slice(3, None, 41)
    want = G.oracle({n: x[:, heads] for n, x in ins.items()}, None)
    G.assert_close(first[0][:, heads].float().cpu().numpy(), want["o"], "o")
    if tangents:
        G.assert_close(first[1][:, heads].float().cpu().numpy(), want["to"], "to")
    assert _lib.device_status() == 0
