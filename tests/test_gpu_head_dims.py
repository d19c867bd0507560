"""bf16 heads of widths other than 64 and 128 on the tcgen05 kernels: the tiles are wider than the head, and the operands
of the second products travel as a 16-bit value plus the rounding of what is left of it."""
import numpy as np
import pytest
import torch

import gpu_util as G
from semicat_b200 import _lib, ops

pytestmark = pytest.mark.gpu

# widths at both ends of the two tiles and in between; lengths at one row, ragged tails and several tiles of each owner
CASES = [(16, 1, 1), (24, 40, 40), (32, 64, 64), (32, 129, 257), (40, 300, 65), (48, 128, 512), (56, 200, 33),
         (72, 130, 97), (96, 128, 256), (96, 257, 31), (120, 1, 300), (120, 384, 129)]


@pytest.mark.parametrize("layout", ["bhld", "bshd", "padded"])
@pytest.mark.parametrize("D,Lq,Lk", CASES)
def test_matches_the_oracle_as_closely_as_the_portable_kernels(D, Lq, Lk, layout):
    """Both families round their results to bf16 once (relative 2-norm error about 2^-9.8); what the operand pairs add,
    about 2^-17 per product, must not show: the error may exceed the portable kernels' by 2 %, and by 1e-6 per element
    where the exact value is zero or cancels (one key: P = 1 and dq is a difference of equal fp32 sums of order 1)."""
    assert ops.selected_kernels(2, 3, Lq, Lk, D) == ops.KERNELS_TCGEN05
    assert ops.selected_kernels(2, 3, Lq, Lk, D, which="bwd") == ops.KERNELS_TCGEN05
    ins = G.rounded(G.synth(2, 3, Lq, Lk, D, seed=D + Lq), torch.bfloat16)
    for mode in ("both", "pri", "tan"):
        want = G.oracle(ins, mode)
        got = G.run(ins, layout=layout, mode=mode)
        simt = G.run(ins, layout=layout, mode=mode, kernels=ops.KERNELS_SIMT)
        G.compare(got, want, mode, f"D={D} {Lq}x{Lk} {layout}")
        for n in got:
            if got[n] is None or n in ("lse", "mu"):
                continue
            floor = 2e-5 * np.linalg.norm(want[n]) + 1e-6 * np.sqrt(want[n].size)
            e, e_simt = (np.linalg.norm(np.asarray(x[n], np.float64) - want[n]) for x in (got, simt))
            assert e <= 1.02 * e_simt + floor, (mode, n, e, e_simt, floor)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("D", [32, 96])
def test_without_tangents(D):
    B, H, L = 2, 3, 161
    ins = G.rounded(G.synth(B, H, L, L, D, seed=3), torch.bfloat16)
    q, k, v = (G.place(ins[n], torch.bfloat16, "bshd") for n in ("q", "k", "v"))
    o = torch.empty_like(q)
    lse = torch.zeros(B, H, ops.stat_len(L), device="cuda")
    ops.jvp_attention_fwd(q, k, v, None, None, None, o, None, lse, None)
    want = G.oracle(ins, "pri")
    G.assert_close(o.float().cpu().numpy(), want["o"], "o")
    G.assert_close(lse[..., :L].cpu().numpy(), want["lse"], "lse")


@pytest.mark.parametrize("D", [16, 40, 64, 96, 128])
def test_forcing_the_selected_family_gives_what_auto_gives(D):
    ins = G.rounded(G.synth(1, 2, 70, 90, D, seed=1), torch.bfloat16)
    assert ops.selected_kernels(1, 2, 70, 90, D) == ops.KERNELS_TCGEN05
    auto, forced = (G.run(ins, kernels=k) for k in (ops.KERNELS_AUTO, ops.KERNELS_TCGEN05))
    assert auto.keys() == forced.keys() and all(np.array_equal(auto[n], forced[n]) for n in auto)


@pytest.mark.parametrize("D,dtype", [(20, torch.bfloat16), (32, torch.float16), (121, torch.bfloat16)])
def test_widths_that_stay_on_the_portable_kernels_cannot_be_forced(D, dtype):
    """Rows that are not 16-byte aligned, and fp16 heads of other widths (their parts lack the exponent range)."""
    assert ops.selected_kernels(1, 1, 64, 64, D, dtype=dtype) == ops.KERNELS_SIMT
    ins = G.rounded(G.synth(1, 1, 64, 64, D, seed=1), dtype)
    with pytest.raises(_lib.JvpAttnError) as e:
        G.run(ins, dtype=dtype, kernels=ops.KERNELS_TCGEN05, mode=None)
    assert e.value.code == -1


@pytest.mark.parametrize("D", [16, 32, 56, 72, 96, 120])
def test_infinite_tangents_come_out_as_from_the_portable_kernels(D):
    """One infinite element of the keys' tangent: scores' tangents, and with them U, are infinite in that column.  The low
    part of an infinite operand is zero, not inf - inf, so infinities and NaN appear where the portable kernels have them."""
    ins = G.rounded(G.synth(2, 2, 70, 90, D, seed=D), torch.bfloat16)
    ins["tk"][:, :, 37, 3] = np.inf
    with np.errstate(invalid="ignore"):
        got, simt = (G.run(ins, mode=None, kernels=k)["to"] for k in (ops.KERNELS_AUTO, ops.KERNELS_SIMT))
    assert np.isinf(simt).any() and np.isnan(simt).any()
    assert np.array_equal(np.isnan(got), np.isnan(simt))
    bad = ~np.isfinite(simt) & ~np.isnan(simt)
    assert np.array_equal(got[bad], simt[bad]) and np.isfinite(got[np.isfinite(simt)]).all()
