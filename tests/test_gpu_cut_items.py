"""How the tensor-core attention kernel spreads calls that do not fill the SMs: single tiles instead of pairs, a last round
taken tile by tile, and key blocks cut into equal runs whose shares are put together behind it.  Against the oracle and,
for the cuts, against the same call without scratch (nothing is cut)."""
import ctypes

import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_masked_prefill import make_mask
from test_gpu_parity import DEV, check, inputs

pytestmark = pytest.mark.gpu


def forward(dtattn, p, scratch):
    s = torch.cuda.current_stream().cuda_stream
    ptr, n = (None, 0) if scratch is None else (scratch.data_ptr(), scratch.numel())
    assert dtattn.lib().dt_sdpa_forward(ctypes.byref(p), ctypes.c_void_p(ptr), n, ctypes.c_void_p(s)) == dtattn.DT_OK
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0


@pytest.mark.parametrize("case", [
    # B, Sq, Sk, Hq, Hkv, D, causal, extra, dtype
    (1, 130, 2000, 4, 2, 64, False, "", torch.float16),        # every item in several runs
    (1, 128, 16384, 1, 1, 128, False, "", torch.bfloat16),     # one item over 32 runs
    (1, 600, 1500, 12, 4, 128, False, "sinks", torch.bfloat16),
    (2, 300, 1700, 8, 4, 256, True, "", torch.bfloat16),       # causal levels of different lengths, head dim 256
    (1, 513, 2900, 4, 1, 256, True, "", torch.float16),        # a last tile of one row
    (1, 1200, 1200, 7, 1, 80, True, "sinks", torch.float16),   # as many keys as queries: the first levels are short
    (1, 2000, 2000, 1, 1, 64, True, "", torch.bfloat16),       # items with fewer key blocks than runs
    (1, 100, 8192, 50, 2, 64, False, "sinks", torch.float16),  # several runs per CTA, the CTAs not all as many
    (1, 100, 8200, 50, 1, 256, True, "", torch.bfloat16),
    (1, 128, 8192, 50, 2, 128, True, "mask", torch.bfloat16),
    (1, 200, 1600, 4, 2, 128, True, "mask", torch.bfloat16),   # masked, aligned rows
    (1, 200, 1601, 4, 2, 64, False, "mask", torch.float16)])   # masked, copied rows
def test_against_the_oracle_and_the_uncut_call(dtattn, case):
    B, Sq, Sk, Hq, Hkv, D, causal, extra, dtype = case
    q, k, v = inputs(B, Sq, Sk, Hq, Hkv, D, dtype, 1601)
    mask = make_mask(1, 1, Sq, Sk, dtype, 1602) if extra == "mask" else None
    if mask is not None:
        mask[..., 5:640] = -torch.finfo(dtype).max  # shares that see next to nothing
    sinks = (so.seeded_normal((Hq,), 1603) * 2).to(dtype) if extra == "sinks" else None
    ref, ref_lse = so.sdpa_explicit(q, k, v, D ** -0.5, causal, mask, compute_dtype=torch.float64, return_lse=True, sinks=sinks)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    out, lse = torch.zeros_like(qd), torch.zeros(B, Hq, Sq, device=DEV)
    md, sd = (None if x is None else x.to(DEV) for x in (mask, sinks))
    p = dtattn.make_params(qd, kd, vd, out, D ** -0.5, causal, md, lse, sinks=sd)
    need = dtattn.workspace_size(p)
    assert need > 4096 + 4 * 32 * 4 * (D + 2), "this case is meant to be cut"
    scratch = torch.full((need,), 0xff, dtype=torch.uint8, device=DEV)
    runs = []
    for _ in range(3):
        out.fill_(float("nan"))
        forward(dtattn, p, scratch)
        runs.append(out.clone())
    check(out, ref.float(), dtype, str(case))
    assert torch.allclose(lse.cpu(), ref_lse.float(), atol=2e-3, rtol=1e-4)
    # the shares are added in the order of the keys
    assert all(torch.equal(r.view(torch.int16), runs[0].view(torch.int16)) for r in runs)
    assert bool((scratch[:4096] == 0xff).all())
    if mask is None:  # (the masked variants cannot run without any scratch)
        forward(dtattn, p, None)
        check(out, ref.float(), dtype, f"{case} uncut")


@pytest.mark.parametrize("where", ["one query row", "a run of keys"])
@pytest.mark.parametrize("extra", ["", "causal", "sinks", "mask"])
@pytest.mark.parametrize("D", [64, 256])
def test_nan_is_kept(dtattn, D, extra, where):
    """A NaN in a query row makes every score of the row NaN, which no maximum shows; NaN keys do so for a whole share.  The
    cut call must give NaN where the uncut one does, and every other row as without the NaN."""
    B, Sq, Sk, Hq, Hkv, dtype = 1, 200, 2304, 4, 2, torch.bfloat16
    q, k, v = (x.to(DEV) for x in inputs(B, Sq, Sk, Hq, Hkv, D, dtype, 1621))
    mask = make_mask(1, 1, Sq, Sk, dtype, 1622).to(DEV) if extra == "mask" else None
    sinks = so.seeded_normal((Hq,), 1623).to(dtype).to(DEV) if extra == "sinks" else None

    def run(scratch_bytes):
        out, lse = torch.zeros_like(q), torch.zeros(B, Hq, Sq, device=DEV)
        p = dtattn.make_params(q, k, v, out, D ** -0.5, extra == "causal", mask, lse, sinks=sinks)
        need = dtattn.workspace_size(p) if scratch_bytes is None else scratch_bytes
        forward(dtattn, p, torch.zeros(need, dtype=torch.uint8, device=DEV) if need else None)
        return out, lse, need

    clean, clean_lse, need = run(None)
    flags_only = 4096 + (((Sq + 31) // 32 * ((Sk + 127) // 128 * 2) + 255) // 256) * 256 if mask is not None else 0
    assert need > 4096 + flags_only, "this case is meant to be cut"
    if where == "one query row":
        q[0, 77, 1, 5] = float("nan")
    else:
        k[0, 256:Sk - 100] = float("nan")  # with the causal rule every row sees some of them
    (cut, cut_lse, _), (whole, whole_lse, _) = run(None), run(flags_only)
    assert bool(whole.isnan().any())
    assert torch.equal(cut.isnan(), whole.isnan()) and torch.equal(cut_lse.isnan(), whole_lse.isnan())
    assert torch.equal(cut_lse == -float("inf"), whole_lse == -float("inf"))
    rows = ~cut.isnan().any(dim=-1)
    assert torch.equal(cut[rows], clean[rows])
    assert torch.equal(cut_lse.transpose(1, 2)[rows], clean_lse.transpose(1, 2)[rows])


@pytest.mark.parametrize("case", [
    # B, Sq, Sk, Hq, Hkv, D, causal, dtype: single tiles throughout (up to 148 of them), and a last round of pairs tile by
    # tile (149 to 222 pairs), with and without a second tile in the last pair
    (1, 300, 200, 40, 8, 64, False, torch.float16), (1, 400, 400, 37, 37, 128, True, torch.bfloat16),
    (1, 1280, 140, 32, 8, 40, False, torch.float16), (1, 1100, 1100, 38, 2, 64, True, torch.bfloat16),
    (2, 900, 70, 20, 20, 128, False, torch.bfloat16),
    # causal: pairs in an odd last round, tiles in an even one
    (1, 600, 600, 55, 5, 40, True, torch.float16), (1, 600, 600, 120, 4, 40, True, torch.float16)])
def test_single_tiles(dtattn, case):
    B, Sq, Sk, Hq, Hkv, D, causal, dtype = case
    q, k, v = inputs(B, Sq, Sk, Hq, Hkv, D, dtype, 1605)
    ref = so.sdpa_explicit(q, k, v, D ** -0.5, causal, compute_dtype=torch.float64)
    out = dtattn.sdpa_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, causal)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    check(out, ref.float(), dtype, str(case))


def test_two_streams_and_a_graph(dtattn):
    """Calls through the Python surface on two streams at once keep their shares apart; a captured call replays."""
    B, Sq, Sk, H, D, dtype = 1, 256, 8192, 4, 128, torch.bfloat16
    cases = []
    for i in range(2):
        q, k, v = (x.to(DEV) for x in inputs(B, Sq, Sk, H, H, D, dtype, 1611 + i))
        cases.append((q, k, v, dtattn.sdpa_forward(q, k, v, D ** -0.5)))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    outs = [[], []]
    for _ in range(20):
        for i, (q, k, v, _) in enumerate(cases):
            with torch.cuda.stream(streams[i]):
                outs[i].append(dtattn.sdpa_forward(q, k, v, D ** -0.5))
    torch.cuda.synchronize()
    for i, (_, _, _, want) in enumerate(cases):
        assert all(torch.equal(o, want) for o in outs[i])
    q, k, v, want = cases[0]
    out = torch.zeros_like(q)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        dtattn.sdpa_forward(q, k, v, D ** -0.5, out=out)
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert dtattn.device_status() == 0
