"""Sparse indexed attention of a few tokens with up to 640 keys each (eight CTAs per token and head group, every key at once)
against the oracle: key counts around its limits, tokens up to and beyond the ones it takes, heads that do not fill a group, with
and without causality, images, views, infinities and NaN."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_sparse_indexed import DEV, ROUND, make_case

pytestmark = pytest.mark.gpu


def few_case(B, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, seed):
    """As make_case, but every token has selected rows: a list per image with "no row" entries in its middle and valid ones at both
    ends.  The ends' rows and the last raw row point where the queries of their KV head do, so that a lost key shows in the output."""
    q, kr, vr, kc, vc, _, sinks = make_case(B, Sq, Sr, Sc, 0, Hq, Hkv, D, dtype, seed)
    g = torch.Generator().manual_seed(seed)
    sel = torch.randint(-2, max(Sc - 1, 1) + 2, (B, Sq, n_sel), generator=g, dtype=torch.int32)
    sel[sel >= Sc - 1] = Sc  # row Sc - 1 is named by the last entry only, row 0 by the first only
    sel[sel == 0] = -1
    loud = q.float().mean(1).reshape(B, Hkv, Hq // Hkv, D).sum(2) * (Sq / (Hq // Hkv)) ** 0.5 * 2
    kr[:, Sr - 1] = loud.to(dtype)
    if n_sel:
        sel[..., 0], sel[..., -1] = 0, Sc - 1
        kc[:, 0] = kc[:, Sc - 1] = loud.to(dtype)
    return q, kr, vr, kc, vc, sel, sinks


def check(dtattn, q, kr, vr, kc, vc, sel, sinks, window, causal=True, same=False):
    """Device tensors; the oracle gets copies of them, with zeros for infinities and NaN (its hidden scores are products too).  Without a
    list there are no compressed rows."""
    D, dtype = q.shape[-1], q.dtype
    if sel.shape[-1] == 0:
        kc = vc = sel = None
    host = [None if t is None else t.cpu() if t is sel else t.cpu().nan_to_num(0, 0, 0) for t in (q, kr, vr, kc, vc, sel)]
    for s in (sinks, None):
        lse = torch.full((q.shape[0], q.shape[2], q.shape[1]), float("nan"), device=DEV)
        out = dtattn.sparse_indexed_attention(q, kr, kr if same else vr, kc, kc if same else vc, sel, D ** -0.5, s, window, causal, lse=lse)
        torch.cuda.synchronize()
        ref, ref_lse = so.sparse_indexed_explicit(host[0], host[1], host[1] if same else host[2], host[3], host[3] if same else host[4],
                                                  host[5], D ** -0.5, None if s is None else s.cpu(), window, causal,
                                                  compute_dtype=torch.float64, return_lse=True)
        mx, mean = so.error_stats(out.float().cpu(), ref.float())
        assert mx <= so.TOL_MAX_ABS + 2 * ROUND[dtype] * float(ref.abs().max()), mx
        assert mean <= so.TOL_MEAN_ABS + ROUND[dtype] * float(ref.abs().mean()), mean
        assert (lse.cpu().double() - ref_lse).abs().max() < 2e-3


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", [
    # Sq, Sr, Sc, n_sel, Hq, Hkv, D, window, values are the keys
    (1, 1, 1, 0, 64, 1, 512, 128, True),       # one key
    (1, 15, 4, 2, 64, 1, 512, 0, True),        # 17 keys: most of the eight CTAs have none
    (1, 300, 75, 0, 64, 1, 512, 128, True),    # 128 keys: 16 per CTA
    (1, 300, 75, 1, 64, 1, 512, 128, True),    # 129
    (2, 3000, 700, 512, 64, 1, 512, 128, True),  # 640, the most it takes
    (1, 3000, 700, 512, 64, 1, 512, 128, True),  # (the decode step)
    (1, 3000, 700, 513, 64, 1, 512, 128, True),  # 641: the other kernel
    (4, 900, 200, 300, 64, 1, 512, 128, True), (5, 900, 200, 300, 64, 1, 512, 128, True),
    (1, 900, 200, 300, 20, 1, 512, 128, True),  # a group of 16 heads and one of 4
    (3, 700, 150, 99, 8, 2, 256, 50, True), (2, 700, 150, 99, 32, 2, 256, 50, False),  # values of their own
    (1, 700, 150, 99, 32, 1, 512, 50, False)])  # (and too wide for two tiles: the other kernel)
def test_few_tokens(dtattn, case, dtype):
    Sq, Sr, Sc, n_sel, Hq, Hkv, D, window, same = case
    t = [x.to(DEV) for x in few_case(1, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, 1801)]
    check(dtattn, *t, window, same=same)
    if n_sel:  # a token whose list names nothing
        t[5][:, 0] = -1
        check(dtattn, *t, window, same=same)


@pytest.mark.parametrize("case", [
    # B, Sq, Hq, D, window, n_sel: token 0 has window + Sq - 1 + n_sel keys
    (2, 2, 64, 512, 64, 62), (2, 2, 64, 512, 64, 63), (2, 2, 64, 512, 64, 64),       # 127, 128, 129
    (2, 2, 64, 512, 128, 510), (2, 2, 64, 512, 128, 511), (2, 2, 64, 512, 128, 512),  # 639, 640, 641 (the other kernel)
    (1, 4, 64, 512, 128, 0), (2, 4, 16, 512, 125, 0), (2, 4, 16, 512, 124, 0),       # 131, 128, 127
    (2, 4, 16, 512, 128, 508), (2, 4, 16, 512, 128, 509), (2, 4, 16, 512, 128, 510),  # 639, 640, 641
    (1, 18, 16, 256, 128, 0), (1, 18, 16, 256, 111, 0), (1, 18, 16, 256, 128, 495), (1, 18, 16, 256, 128, 496)])  # 145, 128, 640, 641
def test_a_window_without_causality(dtattn, case):
    """Every token sees the rows up to the last one, so the first token has the most keys: the window and one per further token."""
    B, Sq, Hq, D, window, n_sel = case
    for Sr in (900, window + Sq // 2):  # (the second: fewer rows than the bound)
        check(dtattn, *[x.to(DEV) for x in few_case(B, Sq, Sr, 200, n_sel, Hq, 1, D, torch.bfloat16, 1811)], window, False, True)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("what", ["q over the images", "q over the tokens", "q over the heads", "keys over the images", "padded rows",
                                  "keys stored by head"])
def test_views_of_every_stride(dtattn, what, causal):
    q, kr, vr, kc, vc, sel, sinks = (x.to(DEV) for x in few_case(2, 3, 300, 70, 90, 32, 2, 256, torch.float16, 1821))
    if what.startswith("q over"):
        axis = ["images", "tokens", "heads"].index(what.split()[-1])
        q = q.narrow(axis, 0, 1).expand(q.shape)
    wide = lambda x: torch.cat([x, x], -1)[..., :256]  # noqa: E731
    view = {"keys over the images": lambda x: x[:1].expand(x.shape), "padded rows": wide,
            "keys stored by head": lambda x: x.transpose(1, 2).contiguous().transpose(1, 2)}.get(what, lambda x: x)
    kr, vr, kc, vc = (view(x) for x in (kr, vr, kc, vc))
    for same in (True, False):
        check(dtattn, q, kr, vr, kc, vc, sel, sinks, 100, causal, same)


@pytest.mark.parametrize("causal", [True, False])
def test_infinities_and_nan(dtattn, causal):
    """In rows that no token names or sees they change nothing; in a row that one head's keys name they reach the tokens that name it; a
    sink of negative infinity is no sink."""
    B, Sq, Sr, Sc, W = 2, 3, 300, 70, 100
    q, kr, vr, kc, vc, sel, sinks = (x.to(DEV) for x in few_case(B, Sq, Sr, Sc, 90, 32, 2, 256, torch.bfloat16, 1831))
    sel[sel == 7] = -1
    sinks[3] = float("-inf")
    for bad in (float("inf"), float("-inf"), float("nan")):
        for x in (kr, vr, kc, vc):
            (x[:, :Sr - Sq - W + 1] if x.shape[1] == Sr else x[:, 7]).fill_(bad)
        for same in (True, False):
            check(dtattn, q, kr, vr, kc, vc, sel, sinks, W, causal, same)
    sel[1, 1, 40] = 7  # NaN in both the row's key and value
    out = dtattn.sparse_indexed_attention(q, kr, vr, kc, vc, sel, 1 / 16, sinks, W, causal)
    nan = out.isnan()
    assert bool(nan[1, 1].all()) and int(nan.sum()) == nan[1, 1].numel()
    kc[:, 7] = 0
    vc[:, 7] = float("inf")  # a weight times infinity
    out = dtattn.sparse_indexed_attention(q, kr, vr, kc, vc, sel, 1 / 16, sinks, W, causal)
    inf = out.isinf()
    assert bool((out[1, 1] == float("inf")).all()) and int(inf.sum()) == inf[1, 1].numel()
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
