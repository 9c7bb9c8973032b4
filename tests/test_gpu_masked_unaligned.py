"""Masks whose rows do not start on 16 bytes (dense [S, S] masks of odd lengths, odd offsets): copied to aligned rows and
served by the tensor-core kernel with two 16-bit parts per weight, against the oracle and the CUDA-core kernel, whose
weights are fp32."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_masked_prefill import make_mask
from test_gpu_parity import DEV, check, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # B, mask batch, mask heads, Sq, Sk, Hq, Hkv, D, causal, dtype: lengths around the 32 x 64 patches and 128-key blocks,
    # every width of the kernel, broadcast and full masks, a mask one element off a 16-byte boundary
    (1, 1, 1, 33, 65, 4, 2, 128, True, torch.bfloat16), (2, 1, 1, 77, 77, 4, 4, 64, False, torch.float16),
    (1, 1, 1, 333, 333, 8, 2, 128, True, torch.bfloat16), (2, 2, 1, 129, 191, 4, 4, 64, False, torch.bfloat16),
    (1, 1, 6, 65, 127, 6, 3, 40, False, torch.float16), (2, 2, 4, 257, 259, 4, 1, 80, True, torch.float16),
    (1, 1, 1, 300, 301, 4, 2, 256, True, torch.bfloat16), (1, 1, 1, 131, 515, 2, 2, 160, False, torch.float16),
    (1, 1, 1, 64, 64, 2, 2, 64, False, torch.bfloat16)])  # (the last one stays on the CUDA cores)
def test_against_oracle_and_cuda_cores(dtattn, case):
    B, bm, hm, Sq, Sk, Hq, Hkv, D, causal, dtype = case
    q, k, v = inputs(B, Sq, Sk, Hq, Hkv, D, dtype, 1401)
    mask = make_mask(bm, hm, Sq, Sk, dtype, 1402)
    mask[..., 3 * Sk // 4:] = mask[..., 3 * Sk // 4:].clamp(max=0) * 0  # a share of the patches holds zeros only
    ref, ref_lse = so.sdpa_explicit(q, k, v, D ** -0.5, causal, mask, compute_dtype=torch.float64, return_lse=True)
    store = torch.zeros(mask.numel() + 1, dtype=dtype, device=DEV)
    shifted = store[1:].view(mask.shape).copy_(mask)  # rows at odd element offsets whatever Sk is
    err = []
    for flags in (0, dtattn.DT_FLAG_FORCE_GENERIC):
        lse = torch.full((B, Hq, Sq), float("nan"), device=DEV)
        out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, causal, shifted, lse=lse, flags=flags)
        torch.cuda.synchronize()
        assert dtattn.device_status() == 0
        check(out, ref.float(), dtype, f"{case} flags={flags}")
        assert torch.allclose(lse.cpu(), ref_lse.float(), atol=2e-3, rtol=1e-4)
        err.append(float((out.cpu().double() - ref).pow(2).mean().sqrt()))
    # both errors are the rounding of the 16-bit result: no precision is given up for the tensor cores
    assert err[0] <= 1.02 * err[1] + 1e-9, err


def test_scratch_limits(dtattn):
    """Without scratch, or with less, the call stays on the CUDA cores; a mask per head whose copy would be larger than
    256 MB asks for none."""
    import ctypes
    B, S, H, D, dtype = 1, 99, 2, 64, torch.float16
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, dtype, 1411))
    mask = make_mask(1, 1, S, S, dtype, 1412).to(DEV)
    want = dtattn.sdpa_forward(q, k, v, D ** -0.5, mask=mask, flags=dtattn.DT_FLAG_FORCE_GENERIC)
    out = torch.zeros_like(q)
    p = dtattn.make_params(q, k, v, out, D ** -0.5, mask=mask)
    need = dtattn.workspace_size(p)
    scratch = torch.full((need,), 0xff, dtype=torch.uint8, device=DEV)
    s = torch.cuda.current_stream().cuda_stream
    for ptr, nbytes in ((None, 0), (scratch.data_ptr(), need - 1), (scratch.data_ptr(), need)):
        out.zero_()
        assert dtattn.lib().dt_sdpa_forward(ctypes.byref(p), ctypes.c_void_p(ptr), nbytes, ctypes.c_void_p(s)) == dtattn.DT_OK
        torch.cuda.synchronize()
        if nbytes < need:
            assert torch.equal(out, want)
        assert float((out.float() - want.float()).abs().max()) < 2e-3
    assert bool((scratch[:4096] == 0xff).all())
    p.Sq = p.Sk = 8201
    p.mask_stride_q, p.mask_stride_h = 8201, 8201 * 8201
    assert dtattn.workspace_size(p) == 0


@pytest.mark.parametrize("what", ["k and v over the heads", "k and v over the batch", "v over the tokens", "q over the batch"])
def test_expanded_views_stay_on_the_cuda_cores(dtattn, what):
    """A view with a zero stride (torch.expand) is not for tensor maps: served as before, whatever scratch there is."""
    B, S, H, D, dtype = 2, 151, 4, 64, torch.bfloat16
    q, k, v = inputs(B, S, S, H, H, D, dtype, 1431)
    if what == "k and v over the heads":
        k, v = k[:, :, :1].expand(B, S, H, D), v[:, :, :1].expand(B, S, H, D)
    elif what == "k and v over the batch":
        k, v = k[:1].expand(B, S, H, D), v[:1].expand(B, S, H, D)
    elif what == "v over the tokens":
        v = v[:, :1].expand(B, S, H, D)
    else:
        q = q[:1].expand(B, S, H, D)
    mask = make_mask(1, 1, S, S, dtype, 1432)
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, False, mask, compute_dtype=torch.float64)

    def dev(t):  # the same view on the device
        small = t[tuple(slice(0, 1) if st == 0 else slice(None) for st in t.stride())]
        return small.to(DEV).expand(t.shape)

    qd, kd, vd = dev(q), dev(k), dev(v)
    out = torch.zeros(B, S, H, D, dtype=dtype, device=DEV)
    dtattn.sdpa_forward(qd, kd, vd, D ** -0.5, mask=mask.to(DEV), out=out)
    want = dtattn.sdpa_forward(qd, kd, vd, D ** -0.5, mask=mask.to(DEV), flags=dtattn.DT_FLAG_FORCE_GENERIC)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, what)
    assert torch.equal(out, want)


@pytest.mark.parametrize("fill", [-1e38, -3e37, -1e4, -float("inf"), "lowest"])
@pytest.mark.parametrize("scale", [0.125, 1.0, 2.0 ** -133])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_fully_masked_rows_and_small_scales(dtattn, dtype, scale, fill):
    """Rows whose every key is masked: an average where the fill stays finite times log2(e), zeros where it does not, as on
    the CUDA cores, whatever the scale is."""
    if dtype == torch.float16 and isinstance(fill, float) and -float("inf") < fill < -65504:
        pytest.skip("not a half-precision number")
    B, S, H, D = 1, 151, 2, 64
    q, k, v = (x.to(DEV) for x in inputs(B, S, S, H, H, D, dtype, 1441))
    mask = make_mask(1, 1, S, S, dtype, 1442).to(DEV)
    mask[..., ::7, :] = -torch.finfo(dtype).max if fill == "lowest" else fill
    mask[..., 3::7, 70:] = -torch.finfo(dtype).max if fill == "lowest" else fill
    got = []
    for flags in (0, dtattn.DT_FLAG_FORCE_GENERIC):
        lse = torch.full((B, H, S), float("nan"), device=DEV)
        got.append((dtattn.sdpa_forward(q, k, v, scale, mask=mask, lse=lse, flags=flags), lse))
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    (out, lse), (want, lse_want) = got
    assert torch.equal(out == 0, want == 0)
    # (the same number before it is rounded, to fp32's precision: at most the neighbouring 16-bit value, one unit in the last place)
    assert float((out.float() - want.float()).abs().max()) <= 2.0 ** (-7 if dtype == torch.bfloat16 else -10) * float(want.abs().max())
    assert torch.equal(lse.isinf(), lse_want.isinf())
    fin = ~lse_want.isinf()
    assert torch.allclose(lse[fin], lse_want[fin], atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("where", ["v", "k", "q"])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("key", [3, 100, 1500])
@pytest.mark.parametrize("case", [(201, 201, True, torch.bfloat16, 64), (130, 2101, False, torch.float16, 128), (77, 2101, True, torch.bfloat16, 256)])
def test_infinities_and_nan(dtattn, case, key, value, where):
    """They reach the rows and columns that they reach on the CUDA cores, bit for bit; the next call is itself again."""
    Sq, Sk, causal, dtype, D = case
    q, k, v = (x.to(DEV) for x in inputs(1, Sq, Sk, 4, 2, D, dtype, 1451))
    x = dict(q=q, k=k, v=v)[where]
    key = min(key, x.shape[1] - 1)
    mask = make_mask(1, 1, Sq, Sk, dtype, 1452).to(DEV)
    clean = dtattn.sdpa_forward(q, k, v, D ** -0.5, causal, mask)
    keep = x[0, key, 1, 5].item()
    x[0, key, 1, 5] = value
    got = []
    for flags in (0, dtattn.DT_FLAG_FORCE_GENERIC):
        lse = torch.full((1, 4, Sq), float("nan"), device=DEV)
        got.append((dtattn.sdpa_forward(q, k, v, D ** -0.5, causal, mask, lse=lse, flags=flags), lse))
    x[0, key, 1, 5] = keep
    again = dtattn.sdpa_forward(q, k, v, D ** -0.5, causal, mask)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    if where == "v":
        assert not bool(got[0][0].isfinite().all())
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.int16 if a.dtype == dtype else torch.int32), b.view(torch.int16 if b.dtype == dtype else torch.int32))
    assert torch.equal(again, clean)


@pytest.mark.parametrize("case", [
    # Sq, Sk, H, D, scratch asked for: either side of the sizes that the CUDA cores keep
    (77, 64, 12, 64, False), (77, 77, 12, 64, False), (100, 127, 4, 40, False), (100, 129, 4, 40, True), (77, 77, 12, 80, True),
    (77, 65, 4, 128, True), (641, 127, 14, 64, True), (640, 127, 14, 64, False)])
def test_which_calls_take_the_tensor_cores(dtattn, case):
    """With the scratch that they ask for, or none, they answer as the CUDA cores do; with less than it bit for bit."""
    import ctypes
    Sq, Sk, H, D, asked = case
    dtype = torch.float16
    q, k, v = (x.to(DEV) for x in inputs(1, Sq, Sk, H, H, D, dtype, 1461))
    store = torch.zeros(Sq * Sk + 1, dtype=dtype, device=DEV)
    mask = store[1:].view(1, 1, Sq, Sk).copy_(make_mask(1, 1, Sq, Sk, dtype, 1462).to(DEV))
    want = dtattn.sdpa_forward(q, k, v, D ** -0.5, mask=mask, flags=dtattn.DT_FLAG_FORCE_GENERIC)
    out = torch.zeros_like(q)
    p = dtattn.make_params(q, k, v, out, D ** -0.5, mask=mask)
    need = dtattn.workspace_size(p)
    assert (need > 0) == asked
    scratch = torch.full((need + 256,), 0xff, dtype=torch.uint8, device=DEV)
    s = torch.cuda.current_stream().cuda_stream
    for ptr, nbytes in ((None, 0), (scratch.data_ptr(), max(need - 1, 0)), (scratch.data_ptr(), need)):
        out.zero_()
        assert dtattn.lib().dt_sdpa_forward(ctypes.byref(p), ctypes.c_void_p(ptr), nbytes, ctypes.c_void_p(s)) == dtattn.DT_OK
        torch.cuda.synchronize()
        assert torch.equal(out, want) or nbytes == need > 0
        assert float((out.float() - want.float()).abs().max()) < 2e-3
    assert bool((scratch[:4096] == 0xff).all()) and bool((scratch[need:] == 0xff).all())
