"""Rows whose maximum grows after an item's first block, in different halves of different blocks, every time, once and not at all: O
is rescaled while the products of the block before may still be running, and waits for them.  Against the oracle."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_parity import DEV, check, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal,window", [(False, 0), (True, 0), (True, 200)])
@pytest.mark.parametrize("D", [40, 64, 128, 256])
@pytest.mark.parametrize("Sq,Sk", [(130, 640), (300, 1000),  # whole blocks; a last block of 104 keys
                                   (300, 160), (300, 161)])  # a second block of 32 and 33 keys
def test_growing_maxima(dtattn, Sq, Sk, D, causal, window, dtype):
    q, k, v = inputs(1, Sq, Sk, 2, 1, D, dtype, 1701)
    # The queries' first dimension against a ramp in the keys' first dimension, one step per 64 keys: row i's scores rise by 2^17 from
    # step to step when i % 3 == 0, fall when i % 3 == 1, and stay as they are otherwise.
    k[0, :, :, 0] = (torch.arange(Sk) // 64 * 1.0).to(dtype)[:, None]
    sign = torch.tensor([1.0, -1.0, 0.0])[torch.arange(Sq) % 3]
    q[0, :, :, 0] = (12.0 * D ** 0.5 * sign).to(dtype)[:, None]
    ref, ref_lse = so.sdpa_explicit(q, k, v, D ** -0.5, causal, compute_dtype=torch.float64, return_lse=True, sliding_window=window)
    lse = torch.full((1, 2, Sq), float("nan"), device=DEV)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, causal, lse=lse, sliding_window=window)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, f"{Sq}x{Sk} D{D} causal={causal} window={window}")
    # a score of up to 180 keeps 24 bits, so its error and the log-sum-exp's is 180 * 2^-24 times a few
    assert torch.allclose(lse.cpu(), ref_lse.float(), atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("peak", [130, 200, 383, 400])
def test_one_late_key_outweighs_all_others(dtattn, peak, D, dtype):
    """A score 30 to 90 above all others (weights of 2^43 to 2^130 against the old reference, beyond what 16 bits or 32 hold) in the
    first or second half of a later block."""
    Sq, Sk = 128, 512
    q, k, v = inputs(1, Sq, Sk, 2, 2, D, dtype, 1711)
    q[..., 0] = (torch.linspace(30, 90, Sq) * D ** 0.5 / 8).to(dtype)[None, :, None]
    k[..., 0] = 0
    k[:, peak, :, 0] = 8
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, compute_dtype=torch.float64)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, f"peak {peak} D{D}")


@pytest.mark.parametrize("D", [40, 64])
@pytest.mark.parametrize("Sq,H", [(300, 80), (300, 60), (500, 80)])  # several rounds, every head ends in a lone tile; one round; pairs only
@pytest.mark.parametrize("Sk", [97, 128, 129, 154, 160, 161])
def test_where_the_order_of_the_products_changes(dtattn, Sk, Sq, H, D):
    """Head dim 64: at one block, and in several rounds with lone last tiles at 160 keys.  Every third row's maximum lies in the second
    block, or in the second half of the only one."""
    q, k, v = inputs(1, Sq, Sk, H, H, D, torch.float16, 1721)
    k[0, :, :, 0] = (torch.arange(Sk) >= min(128, Sk - 20)).half()[:, None]
    q[0, :, :, 0] = (12.0 * D ** 0.5 * torch.tensor([1.0, -1.0, 0.0])[torch.arange(Sq) % 3]).half()[:, None]
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, compute_dtype=torch.float64)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), torch.float16, f"{Sq}x{Sk} H{H} D{D}")
