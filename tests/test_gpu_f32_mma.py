"""fp32 attention on the tensor cores (three bf16 parts per number) against the float64 oracle and the CUDA-core kernel.

The bounds are those of the CUDA-core kernel's own fp32 tests: no accuracy is given up for the tensor cores.
"""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_generic_tiled import check_fp32
from test_gpu_parity import DEV, inputs

pytestmark = pytest.mark.gpu


def both(dtattn, q, k, v, scale, **kw):
    """(tensor cores, CUDA cores) and their log-sum-exps."""
    got = []
    for flags in (0, dtattn.DT_FLAG_FORCE_GENERIC):
        lse = torch.full((q.shape[0], q.shape[2], q.shape[1]), float("nan"), device=DEV)
        out = dtattn.sdpa_forward(q, k, v, scale, lse=lse, flags=flags, **kw)
        torch.cuda.synchronize()
        assert dtattn.device_status() == 0
        got.append((out, lse))
    return got


def rms(x):
    return float(x.double().pow(2).mean().sqrt())


@pytest.mark.parametrize("case", [
    # B, Sq, Sk, Hq, Hkv, D: one tile and one more row, one key block and one more key, odd tails, every width of the
    # kernel (48 / 64 / 80 / 128 columns) at its edges, grouped heads, more work items than SMs
    (1, 128, 128, 1, 1, 8), (1, 129, 129, 2, 1, 40), (2, 300, 257, 8, 8, 40), (1, 511, 385, 4, 2, 48), (1, 200, 143, 3, 3, 56),
    (2, 256, 333, 5, 5, 64), (1, 150, 191, 2, 2, 72), (1, 640, 193, 4, 2, 80), (1, 131, 320, 2, 1, 88), (1, 384, 449, 2, 2, 128),
    (2, 1300, 700, 8, 8, 40), (2, 1300, 700, 8, 8, 80)])
def test_against_the_oracle(dtattn, case):
    B, Sq, Sk, Hq, Hkv, D = case
    q, k, v = inputs(B, Sq, Sk, Hq, Hkv, D, torch.float32, 1301)
    ref, lse_ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, compute_dtype=torch.float64, return_lse=True)
    (out, lse), (out_cc, _) = both(dtattn, q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5)
    check_fp32(out, ref, str(case))
    assert torch.allclose(lse.cpu(), lse_ref.float(), atol=1e-4, rtol=1e-5)
    assert not torch.equal(out, out_cc), "the tensor-core kernel did not run"
    # no less exact than the CUDA-core kernel (a quarter above it allowed for: both errors are random)
    assert rms(out.cpu() - ref.double()) <= 1.25 * rms(out_cc.cpu() - ref.double()) + 1e-8


def test_strided_views_and_outputs(dtattn):
    """q, k, v as slices of one [B, S, 3, H, D] tensor and the output as a slice of a wider one: neighbours stay as they are."""
    B, S, H, D = 2, 260, 4, 40
    qkv = so.seeded_normal((B, S, 3, H, D), 1311)
    ref = so.sdpa_explicit(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], D ** -0.5, False, compute_dtype=torch.float64)
    dev = qkv.to(DEV)
    wide = torch.full((B, S, H + 1, D + 8), 7.0, device=DEV)
    dtattn.sdpa_forward(dev[:, :, 0], dev[:, :, 1], dev[:, :, 2], D ** -0.5, out=wide[:, :, :H, :D])
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check_fp32(wide[:, :, :H, :D], ref, "strided")
    assert bool((wide[:, :, H] == 7.0).all()) and bool((wide[..., D:] == 7.0).all())


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 2.0 ** 58, -3e38, 2.0 ** -111, -1e-38, 1e-44])
@pytest.mark.parametrize("where", ["q", "k", "v"])
def test_values_outside_the_split_range_take_the_cuda_cores(dtattn, value, where):
    B, S, H, D = 1, 300, 2, 64
    t = dict(zip("qkv", (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1321))))
    t[where][0, 170, 1, 5] = value
    (out, lse), (out_cc, lse_cc) = both(dtattn, t["q"], t["k"], t["v"], D ** -0.5)
    assert torch.equal(out.view(torch.int32), out_cc.view(torch.int32)) and torch.equal(lse.view(torch.int32), lse_cc.view(torch.int32))
    t[where][0, 170, 1, 5] = 1.0  # the call behind it is back on the tensor cores
    (out, _), (out_cc, _) = both(dtattn, t["q"], t["k"], t["v"], D ** -0.5)
    assert not torch.equal(out, out_cc) and float((out - out_cc).abs().max()) < 4e-5


def test_large_and_small_magnitudes(dtattn):
    """Scores of some hundreds (one weight per row survives) and values far from 1: relative to the output's size."""
    q, k, v = (x.to(DEV) for x in inputs(1, 256, 300, 2, 2, 64, torch.float32, 1331))
    for fq, fv in ((40.0, 1.0), (1.0, 2.0 ** 50), (1e-3, 2.0 ** -50)):
        ref = so.sdpa_explicit((q * fq).cpu(), k.cpu(), (v * fv).cpu(), 0.125, False, compute_dtype=torch.float64)
        (out, _), (out_cc, _) = both(dtattn, q * fq, k, v * fv, 0.125)
        err, err_cc = rms(out.cpu() - ref.double()), rms(out_cc.cpu() - ref.double())
        assert err <= 1.25 * err_cc + 1e-8 * rms(ref), (fq, fv, err, err_cc)


def test_without_scratch_the_cuda_cores_serve_the_call(dtattn):
    import ctypes
    B, S, H, D = 1, 256, 2, 40
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1341))
    want = dtattn.sdpa_forward(q, k, v, D ** -0.5, flags=dtattn.DT_FLAG_FORCE_GENERIC)
    out = torch.zeros_like(q)
    p = dtattn.make_params(q, k, v, out, D ** -0.5)
    need = dtattn.workspace_size(p)
    assert need > 3 * 6 * q.numel()
    scratch = torch.full((need,), 0xff, dtype=torch.uint8, device=DEV)
    s = torch.cuda.current_stream().cuda_stream
    for ptr, nbytes, same in ((None, 0, True), (scratch.data_ptr(), need - 1, True), (scratch.data_ptr(), need, False)):
        out.zero_()
        assert dtattn.lib().dt_sdpa_forward(ctypes.byref(p), ctypes.c_void_p(ptr), nbytes, ctypes.c_void_p(s)) == dtattn.DT_OK
        torch.cuda.synchronize()
        assert torch.equal(out, want) == same
        assert float((out - want).abs().max()) < 4e-5
    assert bool((scratch[:4096] == 0xff).all())  # the split-KV ticket counters' area


# low 16 bits of the mantissa: all parts of one sign and as large as they get when cut off; the same when rounded
@pytest.mark.parametrize("low", [0xffff, 0x7f3f])
@pytest.mark.parametrize("which", ["q and k", "v", "q, k and v"])
def test_mantissas_with_the_largest_dropped_products(dtattn, which, low):
    """Numbers whose parts are as large as they can be: the partial products left out must not show beside the CUDA-core
    kernel's own roundings."""
    B, S, H, D = 1, 300, 2, 64
    g = torch.Generator().manual_seed(1351)

    def worst(*shape, signs):
        exponent = torch.randint(-2, 2, shape, generator=g, dtype=torch.int32)
        bits = ((exponent + 127) << 23) | low
        x = bits.view(torch.float32)
        return torch.where(torch.rand(shape, generator=g) < 0.5, -x, x) if signs else x

    q, k, v = inputs(B, S, S, H, H, D, torch.float32, 1352)
    if "q" in which:
        q, k = worst(B, S, H, D, signs=True), worst(B, S, H, D, signs=True)
    if "v" in which:
        v = worst(B, S, H, D, signs=False)
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, compute_dtype=torch.float64)
    (out, _), (out_cc, _) = both(dtattn, q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5)
    err, err_cc = rms(out.cpu() - ref.double()), rms(out_cc.cpu() - ref.double())
    assert err <= 1.25 * err_cc + 1e-8 * rms(ref), (which, err, err_cc)


@pytest.mark.parametrize("exponent", [-80, -100, -112, -120, -135])
def test_tiny_values(dtattn, exponent):
    """Values down to the smallest fp32 numbers: relative to the output's size as exact as on the CUDA cores."""
    q, k, v = (x.to(DEV) for x in inputs(1, 200, 300, 2, 2, 64, torch.float32, 1361))
    v = (v.double() * 2.0 ** exponent).float()
    ref = so.sdpa_explicit(q.cpu(), k.cpu(), v.cpu(), 0.125, False, compute_dtype=torch.float64)
    (out, _), (out_cc, _) = both(dtattn, q, k, v, 0.125)
    err, err_cc = rms(out.cpu().double() - ref.double()), rms(out_cc.cpu().double() - ref.double())
    assert err <= 1.25 * err_cc + 1e-8 * rms(ref), (exponent, err, err_cc)
    assert torch.equal(out, out_cc) == (exponent < -80)  # one number below 2^-110 (the smallest of these is 2^-16 of the usual) and it is the CUDA cores' call


def test_scores_beyond_the_fp32_range(dtattn):
    """Scores that overflow once scaled, to either side: the same rows as on the CUDA cores."""
    B, S, H, D = 1, 200, 2, 64
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, torch.float32, 1371))
    q[:, ::3] = 2.0 ** 57
    k[:] = -(2.0 ** 57)
    q[:, 1::3] = -(2.0 ** 57)
    (out, lse), (out_cc, lse_cc) = both(dtattn, q, k, v, 2.0 ** 8)
    assert torch.equal(out.view(torch.int32), out_cc.view(torch.int32)) and torch.equal(lse.view(torch.int32), lse_cc.view(torch.int32))
