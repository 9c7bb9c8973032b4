"""Head dims up to 64, 1024 keys and more, no window, calls that are not cut: the first half of a block's exponentials are taken before its maximum
is known, and again where that turns out to lie far above the maximum so far.  Inputs whose maximum grows again and again, in the
first half of a block, in the second and in both, where rows end in the middle of a block as well.  Against the oracle."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_parity import DEV, check, inputs

pytestmark = pytest.mark.gpu

# what is added to a key's first dimension, by its number (a block has 128 keys)
LEVELS = {
    "second halves": lambda i: i // 64,  # each half above the one before
    "both halves": lambda i: i // 128 * 2,  # (the weights of both count)
    "first halves": lambda i: i // 128 * 2 + (i % 128 < 64),
    "every other block": lambda i: i // 256 * 2 + (i // 128 % 2 == 0) * 0.5,
}


def rising(Sq, Sk, Hq, Hkv, D, dtype, level, seed):
    """Row i's scores rise by 12, 2^17 in its weights, from one level to the next when i % 3 == 0, fall when i % 3 == 1, and stay when i % 3 == 2."""
    q, k, v = inputs(1, Sq, Sk, Hq, Hkv, D, dtype, seed)
    k[0, :, :, 0] = (LEVELS[level](torch.arange(Sk)) * 1.0).to(dtype)[:, None]
    sign = torch.tensor([1.0, -1.0, 0.0])[torch.arange(Sq) % 3]
    q[0, :, :, 0] = (12.0 * D ** 0.5 * sign).to(dtype)[:, None]
    return q, k, v


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [40, 64])
@pytest.mark.parametrize("Sk,H", [(1024, 26), (1025, 52), (1129, 26), (1300, 52)])  # 78 single tiles; pairs and a lone tile per head
@pytest.mark.parametrize("level", sorted(LEVELS))
def test_growing_maxima(dtattn, Sk, H, D, causal, dtype, level):
    Sq = 300
    q, k, v = rising(Sq, Sk, H, H // 2, D, dtype, level, 1901)
    ref, ref_lse = so.sdpa_explicit(q, k, v, D ** -0.5, causal, compute_dtype=torch.float64, return_lse=True)
    lse = torch.full((1, H, Sq), float("nan"), device=DEV)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, causal, lse=lse)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, f"{Sq}x{Sk} H{H} D{D} causal={causal} {level}")
    # a score of up to 240 keeps 24 bits, so its error and the log-sum-exp's is 240 * 2^-24 times a few
    assert torch.allclose(lse.cpu(), ref_lse.float(), atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [40, 64])
@pytest.mark.parametrize("peak", [129, 200, 1023, 1024, 1128])
def test_one_late_key_outweighs_all_others(dtattn, peak, D, dtype):
    """A score 30 to 90 above all others: weights of 2^43 to 2^130 against the maximum so far, beyond what 16 bits or 32 hold, in either half of a
    block that is whole, the last one, or of one key less."""
    Sq, Sk, H = 300, 1129, 26
    q, k, v = inputs(1, Sq, Sk, H, H, D, dtype, 1911)
    q[..., 0] = (torch.linspace(30, 90, Sq) * D ** 0.5 / 8).to(dtype)[None, :, None]
    k[..., 0] = 0
    k[:, peak, :, 0] = 8
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, compute_dtype=torch.float64)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, f"peak {peak} D{D}")


@pytest.mark.parametrize("level", ["both halves", "first halves"])
def test_sequences_of_different_lengths(dtattn, level):
    """One of them of 1024 keys or more decides for all of them, down to one of a single key."""
    lengths, H, D, dtype = [1100, 1, 40, 129, 1300, 300], 4, 64, torch.bfloat16
    off = [0]
    for n in lengths:
        off.append(off[-1] + n)
    q, k, v = (torch.cat(t, dim=1) for t in zip(*(rising(n, n, H, H, D, dtype, level, 1921 + 10 * i) for i, n in enumerate(lengths))))
    offsets = torch.tensor(off, dtype=torch.int32, device=DEV)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, seq_offsets_q=offsets, seq_offsets_k=offsets,
                              max_seq_q=max(lengths), max_seq_k=max(lengths))
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    for a, b in zip(off, off[1:]):
        ref = so.sdpa_explicit(q[:, a:b], k[:, a:b], v[:, a:b], D ** -0.5, False, compute_dtype=torch.float64)
        check(out[:, a:b], ref.float(), dtype, f"rows {a} to {b}")
