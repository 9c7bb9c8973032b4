"""Sparse indexed attention of many tokens (the tcgen05 kernel: 64 heads per KV head, values = keys, head dim 256 or 512)
against the oracle, at the edges of its 48-key tiles, its head groups and its dispatch."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_parity import DEV
from test_gpu_sparse_indexed import ROUND, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # B, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, window, sinks, causal
    (1, 16, 64, 0, 0, 64, 1, 512, torch.bfloat16, 48, True, True),      # one tile at most, the smallest dispatched count
    (1, 70, 120, 30, 1, 64, 1, 512, torch.float16, 48, True, True),     # one key more than a tile
    (1, 150, 300, 64, 48, 64, 1, 512, torch.bfloat16, 128, True, True),  # more tokens than SMs: a second token per CTA
    (1, 320, 500, 90, 200, 64, 1, 512, torch.float16, 128, False, True),  # lists longer than the rows, no sinks, third tokens
    (2, 70, 100, 40, 33, 128, 1, 512, torch.bfloat16, 0, True, True),   # two head groups, batch, no window
    (1, 40, 90, 25, 60, 128, 2, 256, torch.float16, 20, True, True),    # two KV heads, head dim 256
    (1, 80, 100, 16, 16, 64, 1, 256, torch.bfloat16, 0, True, False),   # every token sees every raw row
    (1, 18, 700, 50, 60, 64, 1, 256, torch.float16, 128, True, True),   # either side of the dispatch at head dim 256
    (1, 19, 700, 50, 60, 64, 1, 256, torch.float16, 128, True, True),
])
def test_against_the_oracle(dtattn, case):
    B, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, window, with_sinks, causal = case
    q, kr, _, kc, _, sel, sinks = make_case(B, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, 1501, per_batch_lists=B > 1)
    if not with_sinks:
        sinks = None
    if n_sel:
        sel[:, 3] = -1  # a token without any selected row
    ref, ref_lse = so.sparse_indexed_explicit(q, kr, kr, kc if Sc else None, kc if Sc else None, sel if n_sel else None, D ** -0.5,
                                              sinks, window, compute_dtype=torch.float64, return_lse=True, is_causal=causal)
    rd, cd = kr.to(DEV), kc.to(DEV) if Sc else None
    wide = torch.full((B, Sq, Hq, D + 64), 7.0, dtype=dtype, device=DEV)
    lse = torch.full((B, Hq, Sq), float("nan"), device=DEV)
    out = dtattn.sparse_indexed_attention(q.to(DEV), rd, rd, cd, cd, sel.to(DEV) if n_sel else None, D ** -0.5,
                                          None if sinks is None else sinks.to(DEV), window, is_causal=causal, out=wide[..., :D], lse=lse)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    got = out.float().cpu()
    assert torch.isfinite(got).all() and bool((wide[..., D:] == 7.0).all())
    mx, mean = so.error_stats(got, ref.float())
    assert mx <= so.TOL_MAX_ABS + 2 * ROUND[dtype] * float(ref.abs().max()), (case, mx)
    assert mean <= so.TOL_MEAN_ABS + ROUND[dtype] * float(ref.abs().mean()), (case, mean)
    assert (lse.cpu().double() - ref_lse).abs().max() < 2e-3


def test_growing_scores_and_hidden_tokens(dtattn):
    """Keys ordered so that every tile raises each head's maximum by more than the rescale threshold, and tokens that see
    nothing at all (zeros without sinks)."""
    B, Sq, Sr, Hq, D, dtype = 1, 66, 400, 64, 512, torch.bfloat16
    q = torch.ones(B, Sq, Hq, D, dtype=dtype) * 0.25
    kr = (torch.linspace(0.01, 3.0, Sr).view(1, Sr, 1, 1) * torch.ones(D)).to(dtype) + so.seeded_normal((1, Sr, 1, D), 1511).to(dtype) * 0.1
    ref = so.sparse_indexed_explicit(q, kr, kr, None, None, None, 1.0, None, 350, compute_dtype=torch.float64)
    out = dtattn.sparse_indexed_attention(q.to(DEV), kr.to(DEV), (d := kr.to(DEV)), None, None, None, 1.0, None, 350)
    same = dtattn.sparse_indexed_attention(q.to(DEV), d, d, None, None, None, 1.0, None, 350)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    for got in (out, same):
        assert float((got.float().cpu() - ref.float()).abs().max()) <= 2 * ROUND[dtype] * float(ref.abs().max()) + so.TOL_MAX_ABS
    sel = torch.full((1, Sq, 5), -1, dtype=torch.int32, device=DEV)
    comp = torch.full((1, 7, 1, D), float("nan"), dtype=dtype, device=DEV)  # rows nobody names are never used
    empty = torch.zeros(1, 1, 1, D, dtype=dtype, device=DEV)[:, :0]
    got = dtattn.sparse_indexed_attention(q.to(DEV), empty, empty, comp, comp, sel, 1.0, None, 128)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0 and bool((got == 0).all())


@pytest.mark.parametrize("amplitude", [1.0, 4.0])  # weights spread over many keys; a few keys with most of the weight
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_weights_are_not_rounded_to_16_bits(dtattn, dtype, amplitude):
    """Error against 64 bits no larger than the CUDA-core kernel's, whose weights are fp32: both are the rounding of the
    16-bit result (2 % for its random part).  Weights of 16 bits show 1.2 to 1.3 times that."""
    B, Sq, Sr, Sc, n_sel, H, D = 1, 48, 700, 160, 300, 64, 512
    q, kr, _, kc, _, sel, sinks = make_case(B, Sq, Sr, Sc, n_sel, H, 1, D, dtype, 1521)
    q = (q.float() * amplitude).to(dtype)
    ref = so.sparse_indexed_explicit(q, kr, kr, kc, kc, sel, D ** -0.5, sinks, 128, compute_dtype=torch.float64)
    rd, cd = kr.to(DEV), kc.to(DEV)
    err = []
    for flags in (0, dtattn.DT_FLAG_FORCE_GENERIC):
        out = dtattn.sparse_indexed_attention(q.to(DEV), rd, rd, cd, cd, sel.to(DEV), D ** -0.5, sinks.to(DEV), 128, flags=flags)
        torch.cuda.synchronize()
        assert dtattn.device_status() == 0
        err.append(float((out.cpu().double() - ref).norm() / ref.norm()))
    assert err[0] <= 1.02 * err[1], err


@pytest.mark.parametrize("n_keys", [20, 48, 70, 96, 97, 200, 430])
def test_many_short_tokens_per_cta(dtattn, n_keys):
    """Every CTA takes several tokens of one, two and more 48-key tiles one after another: a token's end and the next one's
    first tiles overlap.  Repeated, bit for bit the same."""
    Sq, Sr, H, D, dtype = 620, 1060, 64, 256, torch.bfloat16
    q = so.seeded_normal((1, Sq, H, D), 1531).to(dtype) * 3
    kr = so.seeded_normal((1, Sr, 1, D), 1532).to(dtype)
    ref = so.sparse_indexed_explicit(q, kr, kr, None, None, None, D ** -0.5, None, n_keys, compute_dtype=torch.float64)
    qd, rd = q.to(DEV), kr.to(DEV)
    outs = [dtattn.sparse_indexed_attention(qd, rd, rd, None, None, None, D ** -0.5, None, n_keys) for _ in range(5)]
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    assert float((outs[0].float().cpu() - ref.float()).abs().max()) <= 2 * ROUND[dtype] * float(ref.abs().max()) + so.TOL_MAX_ABS
    assert all(torch.equal(o, outs[0]) for o in outs)


@pytest.mark.parametrize("what", ["q over the batch", "q over the tokens", "q over the heads", "keys over the batch", "keys over the KV heads",
                                  "keys stored by head", "lone key row"])
def test_views_of_every_stride(dtattn, what):
    """Views that tensor maps do not describe (an expanded axis has stride 0) and unusual ones that they may: as the oracle."""
    B, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype = 2, 40, 90, 30, 20, 128, 2, 256, torch.bfloat16
    if what == "lone key row":
        Sr, Sc = 60, 1
    q, kr, _, kc, _, sel, sinks = make_case(B, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, 1541, per_batch_lists=True)
    axis = {"q over the batch": (0, 0), "q over the tokens": (0, 1), "q over the heads": (0, 2), "keys over the batch": (1, 0),
            "keys over the KV heads": (1, 2)}.get(what)
    if axis is not None:
        one = lambda t: t.narrow(axis[1], 0, 1).contiguous().to(DEV).expand(t.shape)  # noqa: E731
    if axis is not None and axis[0] == 0:
        qd, rd, cd = one(q), kr.to(DEV), kc.to(DEV)
    elif axis is not None:
        qd, rd, cd = q.to(DEV), one(kr), one(kc)
    elif what == "keys stored by head":
        qd, rd, cd = q.to(DEV), kr.to(DEV).transpose(1, 2).contiguous().transpose(1, 2), kc.to(DEV).transpose(1, 2).contiguous().transpose(1, 2)
    else:
        qd, rd, cd = q.to(DEV), kr.to(DEV), kc.to(DEV)
    ref = so.sparse_indexed_explicit(qd.cpu(), rd.cpu(), rd.cpu(), cd.cpu(), cd.cpu(), sel, D ** -0.5, sinks, 40, compute_dtype=torch.float64)
    out = torch.zeros(B, Sq, Hq, D, dtype=dtype, device=DEV)
    dtattn.sparse_indexed_attention(qd, rd, rd, cd, cd, sel.to(DEV), D ** -0.5, sinks.to(DEV), 40, out=out)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    mx, mean = so.error_stats(out.float().cpu(), ref.float())
    assert mx <= so.TOL_MAX_ABS + 2 * ROUND[dtype] * float(ref.abs().max()), (what, mx)
    assert mean <= so.TOL_MEAN_ABS + ROUND[dtype] * float(ref.abs().mean()), (what, mean)
