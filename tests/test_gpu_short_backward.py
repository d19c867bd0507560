"""Backward of sequences within one tile (one CTA per (batch, head) pair): lengths at the edges of the tile and of the 16-row
steps, one or many pairs per CTA, each set of cotangents, against the fp64 oracle and the canaries around every output."""
import pytest
import torch

import gpu_util as G
from semicat_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["both", "tan", "pri"])
@pytest.mark.parametrize("B,H,Lq,Lk,dtype,layout", [
    (4, 4, 128, 128, torch.bfloat16, "bshd"), (5, 7, 1, 128, torch.bfloat16, "padded"), (16, 1, 128, 1, torch.float16, "bhld"),
    (2, 8, 1, 1, torch.bfloat16, "bshd"), (3, 6, 63, 65, torch.bfloat16, "bshd"), (2, 9, 127, 33, torch.float16, "padded"),
    (3, 8, 17, 112, torch.bfloat16, "bhld"), (41, 12, 100, 128, torch.bfloat16, "bshd"), (2, 7, 64, 64, torch.bfloat16, "bshd")])
def test_gradients(B, H, Lq, Lk, dtype, layout, mode):
    ins = G.rounded(G.synth(B, H, Lq, Lk, 64, seed=Lq + 3 * Lk), dtype)
    got = G.run(ins, dtype=dtype, layout=layout, mode=mode)
    want = G.oracle(ins, mode)
    for n in G.GRAD_NAMES:
        if n in got:
            G.assert_close(got[n], want[n], n)
    assert _lib.device_status() == 0


def test_replays_are_equal():
    """Many replays back to back, three pairs per CTA: every wait meets its own phase."""
    ins = G.rounded(G.synth(20, 24, 128, 128, 64, seed=2), torch.bfloat16)
    t = {n: G.place(ins[n], torch.bfloat16, "bshd") for n in (*G.IN_NAMES, "g_o", "g_od")}
    o, to = torch.empty_like(t["q"]), torch.empty_like(t["q"])
    lse = torch.zeros(20, 24, ops.stat_len(128), device="cuda")
    mu = torch.zeros_like(lse)
    for tang in (True, False):
        grads = [torch.full_like(t[n], G.CANARY) for n in G.IN_NAMES]
        plan = ops.Plan(*[t[n] for n in G.IN_NAMES], o, to, lse, mu, g_o=t["g_o"], g_to=t["g_od"] if tang else None, grads=grads)
        plan.forward()
        plan.backward()
        first = [g.clone() for g in grads]
        for _ in range(200):
            plan.backward()
        assert all(torch.equal(a, b) for a, b in zip(first, grads))
    assert _lib.device_status() == 0
