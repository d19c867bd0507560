"""Attention without tangents at the edges of its tiles: the instances that share an SM (forward three CTAs, backward two at
head_dim 64) and the one-CTA ones, against the fp64 oracle."""
import pytest
import torch

import gpu_util as G
from semicat_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Lq,Lk,D,dtype", [
    (1, 1, 1, 1, 64, torch.bfloat16), (2, 3, 64, 65, 64, torch.bfloat16), (2, 3, 127, 129, 64, torch.float16),
    (1, 2, 700, 333, 64, torch.bfloat16), (32, 12, 128, 128, 64, torch.bfloat16), (1, 2, 129, 1, 64, torch.bfloat16),
    (1, 1, 1, 130, 128, torch.bfloat16), (2, 3, 257, 190, 128, torch.float16), (2, 80, 128, 64, 128, torch.bfloat16),
    (2, 3, 200, 129, 40, torch.bfloat16), (2, 3, 65, 300, 96, torch.bfloat16)])
def test_forward_and_backward(B, H, Lq, Lk, D, dtype):
    ins = G.rounded(G.synth(B, H, Lq, Lk, D, seed=Lq + Lk), dtype)
    q, k, v, g = (G.place(ins[n], dtype, "bshd") for n in ("q", "k", "v", "g_o"))
    buf, o, pad, n = G.guarded_like(q)
    lse = torch.full((B, H, ops.stat_len(Lq)), G.CANARY, device="cuda")
    ops.jvp_attention_fwd(q, k, v, None, None, None, o, None, lse, None)
    guards = [G.guarded_like(x) for x in (q, k, v)]
    ops.jvp_attention_bwd(q, k, v, None, None, None, o, None, g, None, lse, None, *[x[1] for x in guards])
    torch.cuda.synchronize()
    want = G.oracle(ins, "pri")
    G.check_canaries(buf, pad, n, "o")
    assert bool((lse[..., Lq:] == G.CANARY).all())
    G.assert_close(o.float().cpu().numpy(), want["o"], "o")
    G.assert_close(lse[..., :Lq].cpu().numpy(), want["lse"], "lse", rtol=1e-3, atol=2e-3)
    for name, (b_, view, p_, n_) in zip(("dq", "dk", "dv"), guards):
        G.check_canaries(b_, p_, n_, name)
        G.assert_close(view.float().cpu().numpy(), want[name], name)
    assert _lib.device_status() == 0
