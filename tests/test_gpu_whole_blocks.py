"""Prefill calls around the lengths where whole blocks of 128 keys take a path of their own: blocks that end in 1, 32 and 33 keys behind
one, two and three whole ones, a causal diagonal and a window's edge inside whole blocks, an additive mask.  Against the oracle."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_parity import DEV, check, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "causal", "window", "mask"])
@pytest.mark.parametrize("D", [64, 80, 128, 256])
@pytest.mark.parametrize("Sk", [160, 161, 257, 288, 289, 384, 385, 512, 641])
def test_against_the_oracle(dtattn, Sk, D, form):
    Sq, dtype = 150, torch.bfloat16
    q, k, v = inputs(1, Sq, Sk, 4, 2, D, dtype, 1801)
    causal, window, mask = form in ("causal", "window"), 131 if form == "window" else 0, None
    if form == "mask":
        mask = torch.zeros(1, 1, Sq, (Sk + 7) // 8 * 8, dtype=dtype)[..., :Sk]  # (rows start on 16 bytes)
        mask[..., Sk - 40:] = -torch.finfo(dtype).max
        mask[..., 70, :] = 1.5
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, causal, mask=mask, compute_dtype=torch.float64, sliding_window=window)
    dev_mask = None
    if mask is not None:
        dev_mask = torch.zeros(1, 1, Sq, (Sk + 7) // 8 * 8, dtype=dtype, device=DEV)[..., :Sk]
        dev_mask.copy_(mask)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, causal, mask=dev_mask, sliding_window=window)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, f"{Sq}x{Sk} D{D} {form}")
