"""fp32 attention on the tensor cores in calls of more tiles than SMs, and inputs that no part of a number may be left out of: weights of one,
weights that are small beside one whose value is zero, values of very different sizes.  Against the float64 oracle.

Bounds: the CUDA-core kernel's own fp32 error, or one that is derived beside the test.
"""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_f32_mma import both, rms
from test_gpu_generic_tiled import check_fp32
from test_gpu_parity import DEV, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # B, Sq, Sk, Hq, Hkv, D, all of more tiles than SMs: widths at their edges, heads that end in a tile of one row, key blocks that
    # end in 1, 16, 64, 65 and 128 keys, grouped heads
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


def aimed(k, target):
    """Queries that see one key each (the next one's weight is below e^-100): that key, over its own square, times 4000."""
    x = k[:, target]
    return 4000.0 * x / x.pow(2).sum(dim=-1, keepdim=True)


@pytest.mark.parametrize("D", [40, 64])
def test_one_weight_of_one(dtattn, D):
    """Nothing is added up, so the output is V but for the roundings of weight times V, of one over the weight and of the result: 2^-24 of it each, or
    2^-23 cut off, whose root mean squares, a third of them each, add up to less than 2^-23."""
    B, S, H = 1, 600, 40
    _, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1441))
    k /= k.pow(2).mean(dim=-1, keepdim=True).sqrt()
    target = torch.randperm(S, generator=torch.Generator().manual_seed(1442)).to(DEV)
    out = dtattn.sdpa_forward(aimed(k, target), k, v, D ** -0.5)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    assert rms(out.double() - v[:, target].double()) <= 2.0 ** -23 * rms(v)


@pytest.mark.parametrize("D", [40, 64])
@pytest.mark.parametrize("gap", [14.0, 20.0, 27.0, 60.0])
def test_the_heaviest_key_adds_nothing(dtattn, gap, D):
    """A key `gap` above all others whose V is zero: what the others add, relative to its own size.  A weight is exp2 of a difference of two
    numbers of gap * log2(e), each with a rounding of 2^-24 of it (the scale's and the product's): gap * 2^-23 of the weight."""
    B, S, H = 1, 600, 40
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1451))
    q[..., 0], k[..., 0] = D ** 0.5, 0.0
    k[:, 77] = 0.0
    k[:, 77, :, 0] = gap
    v[:, 77] = 0.0
    ref = so.sdpa_explicit(q.cpu(), k.cpu(), v.cpu(), D ** -0.5, False, compute_dtype=torch.float64)
    (out, lse), (out_cc, lse_cc) = both(dtattn, q, k, v, D ** -0.5)
    err, err_cc = rms(out.cpu() - ref.double()), rms(out_cc.cpu() - ref.double())
    assert err <= max(err_cc, gap * 2.0 ** -23 * rms(ref)), (gap, err / rms(ref), err_cc / rms(ref))
    assert torch.allclose(lse, lse_cc, atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("per_block", [1, 8, 15])
def test_a_few_small_values_among_zeros(dtattn, per_block):
    """A column of V that is zero but for some numbers far below the other columns', as exact relative to its own size as on the CUDA cores."""
    B, S, H, D = 1, 600, 40, 40
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1461))
    keep = torch.arange(S, device=DEV) % 128 < per_block
    v[..., 5] *= 2.0 ** -30
    v[:, ~keep, :, 5] = 0.0
    ref = so.sdpa_explicit(q.cpu(), k.cpu(), v.cpu(), D ** -0.5, False, compute_dtype=torch.float64)
    (out, _), (out_cc, _) = both(dtattn, q, k, v, D ** -0.5)
    for d in (0, 5):
        e, e_cc = rms(out[..., d].cpu() - ref[..., d].double()), rms(out_cc[..., d].cpu() - ref[..., d].double())
        assert e <= 1.25 * e_cc + 1e-8 * rms(ref[..., d]), (d, e / rms(ref[..., d]), e_cc / rms(ref[..., d]))


@pytest.mark.parametrize("where", ["a column", "rows", "one head's last rows", "all but one number", "all numbers"])
def test_values_of_very_different_sizes(dtattn, where):
    """Numbers of V far below others of their block, each column as exact relative to its own size as on the CUDA cores; a third of the queries see one
    key each, the small ones among them, and a row's output is as exact relative to its own size."""
    B, S, H, D = 1, 600, 40, 64
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1471))
    q[:, ::3] = aimed(k, torch.arange(0, S, 3, device=DEV) * 7 % S)
    if where == "a column":
        v[..., 5] *= 2.0 ** -24
    elif where == "rows":
        v[:, ::7] *= 2.0 ** -22
    elif where == "one head's last rows":
        v[:, 590:, 3] *= 2.0 ** -30
    elif where == "all but one number":
        v *= 2.0 ** -24
        v[:, 100, :, 9] = 1.0
    else:
        v *= 2.0 ** -60
    ref = so.sdpa_explicit(q.cpu(), k.cpu(), v.cpu(), D ** -0.5, False, compute_dtype=torch.float64).double()
    (out, lse), (out_cc, lse_cc) = both(dtattn, q, k, v, D ** -0.5)
    size = ref.pow(2).mean(dim=-1, keepdim=True).sqrt()  # of each row
    e, e_cc = rms((out.cpu() - ref) / size), rms((out_cc.cpu() - ref) / size)
    assert e <= 1.25 * e_cc + 1e-8, (where, e, e_cc)
    for d in (0, 5, 63):
        e, e_cc = rms(out[..., d].cpu() - ref[..., d]), rms(out_cc[..., d].cpu() - ref[..., d])
        assert e <= 1.25 * e_cc + 1e-8 * rms(ref[..., d]), (where, d, e, e_cc)
    assert torch.allclose(lse, lse_cc, atol=1e-4, rtol=1e-5)
