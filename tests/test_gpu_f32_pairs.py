"""fp32 attention with two query tiles to a CTA (weights and V as two fp16 parts) against the float64 oracle.

Bounds: the CUDA-core kernel's own fp32 error, as for the kernel with one tile to a CTA.
"""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_f32_mma import both, rms
from test_gpu_generic_tiled import check_fp32
from test_gpu_parity import DEV, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # B, Sq, Sk, Hq, Hkv, D, all of more single tiles than SMs: both widths of the kernel at their edges, heads that end in a lone tile
    # (300 rows: three), in a tile of one row, in whole pairs; key blocks that end in 1, 16, 64, 65 and 128 keys; grouped heads; two rounds of pairs
    (1, 300, 513, 64, 64, 40), (1, 385, 528, 48, 16, 40), (2, 256, 576, 80, 80, 48), (1, 257, 577, 64, 8, 56), (2, 300, 640, 32, 32, 64),
    (1, 512, 897, 100, 20, 40), (1, 512, 1024, 100, 100, 64)])
def test_against_the_oracle(dtattn, case):
    B, Sq, Sk, Hq, Hkv, D = case
    q, k, v = inputs(B, Sq, Sk, Hq, Hkv, D, torch.float32, 1401)
    ref, lse_ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, compute_dtype=torch.float64, return_lse=True)
    (out, lse), (out_cc, _) = both(dtattn, q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5)
    check_fp32(out, ref, str(case))
    assert torch.allclose(lse.cpu(), lse_ref.float(), atol=1e-4, rtol=1e-5)
    assert not torch.equal(out, out_cc), "the tensor-core kernel did not run"
    assert rms(out.cpu() - ref.double()) <= 1.25 * rms(out_cc.cpu() - ref.double()) + 1e-8


def test_strided_views_and_outputs(dtattn):
    B, S, H, D = 1, 600, 40, 40
    qkv = so.seeded_normal((B, S, 3, H, D), 1411)
    ref = so.sdpa_explicit(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], D ** -0.5, False, compute_dtype=torch.float64)
    dev = qkv.to(DEV)
    wide = torch.full((B, S, H + 1, D + 8), 7.0, device=DEV)
    dtattn.sdpa_forward(dev[:, :, 0], dev[:, :, 1], dev[:, :, 2], D ** -0.5, out=wide[:, :, :H, :D])
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check_fp32(wide[:, :, :H, :D], ref, "strided")
    assert bool((wide[:, :, H] == 7.0).all()) and bool((wide[..., D:] == 7.0).all())


@pytest.mark.parametrize("where", ["a column", "rows", "one head's last rows", "everything small"])
def test_values_that_two_fp16_parts_do_not_hold(dtattn, where):
    """V with numbers far below their block's largest, which the kernel with one tile to a CTA computes behind the pass that finds
    them: each column as exact, relative to its own size, as on the CUDA cores."""
    B, S, H, D = 1, 600, 40, 64
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1421))
    if where == "a column":
        v[..., 5] *= 2.0 ** -24
    elif where == "rows":
        v[:, ::7] *= 2.0 ** -22
    elif where == "one head's last rows":
        v[:, 590:, 3] *= 2.0 ** -30
    else:
        v *= 2.0 ** -60
    ref = so.sdpa_explicit(q.cpu(), k.cpu(), v.cpu(), D ** -0.5, False, compute_dtype=torch.float64)
    (out, _), (out_cc, _) = both(dtattn, q, k, v, D ** -0.5)
    assert not torch.equal(out, out_cc)
    for d in (0, 5, 63):
        e, e_cc = rms(out[..., d].cpu() - ref[..., d].double()), rms(out_cc[..., d].cpu() - ref[..., d].double())
        assert e <= 1.25 * e_cc + 1e-8 * rms(ref[..., d]), (where, d, e, e_cc)


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 2.0 ** 58, 2.0 ** -111])
@pytest.mark.parametrize("where", ["q", "k", "v"])
def test_values_outside_the_split_range_take_the_cuda_cores(dtattn, value, where):
    B, S, H, D = 1, 600, 40, 40
    t = dict(zip("qkv", (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1431))))
    t[where][0, 170, 1, 5] = value
    (out, lse), (out_cc, lse_cc) = both(dtattn, t["q"], t["k"], t["v"], D ** -0.5)
    assert torch.equal(out.view(torch.int32), out_cc.view(torch.int32)) and torch.equal(lse.view(torch.int32), lse_cc.view(torch.int32))
    t[where][0, 170, 1, 5] = 1.0  # the call behind it is back on the tensor cores
    (out, _), (out_cc, _) = both(dtattn, t["q"], t["k"], t["v"], D ** -0.5)
    assert not torch.equal(out, out_cc) and float((out - out_cc).abs().max()) < 4e-5
