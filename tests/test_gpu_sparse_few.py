"""Sparse indexed attention of a few tokens with up to 640 keys each (eight CTAs per token and head group, every key at once)
against the oracle: key counts around its limits, tokens up to and beyond the ones it takes, heads that do not fill a group."""
import pytest
import torch

from oracle import sdpa_oracle as so
from test_gpu_sparse_indexed import DEV, ROUND, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", [
    # Sq, Sr, Sc, n_sel, Hq, Hkv, D, window, values are the keys
    (1, 1, 1, 0, 64, 1, 512, 128, True),       # one key
    (1, 15, 4, 2, 64, 1, 512, 0, True),        # 17 keys: most of the eight CTAs have none
    (1, 300, 75, 0, 64, 1, 512, 128, True),    # 128 keys: 16 per CTA
    (1, 300, 75, 1, 64, 1, 512, 128, True),    # 129
    (2, 3000, 700, 512, 64, 1, 512, 128, True),  # 640, the most it takes
    (1, 3000, 700, 513, 64, 1, 512, 128, True),  # 641: the other kernel
    (4, 900, 200, 300, 64, 1, 512, 128, True), (5, 900, 200, 300, 64, 1, 512, 128, True),
    (1, 900, 200, 300, 20, 1, 512, 128, True),  # a group of 16 heads and one of 4
    (3, 700, 150, 99, 8, 2, 256, 50, True), (2, 700, 150, 99, 32, 2, 256, 50, False),  # values of their own
    (1, 700, 150, 99, 32, 1, 512, 50, False)])  # (and too wide for two tiles: the other kernel)
def test_few_tokens(dtattn, case, dtype):
    Sq, Sr, Sc, n_sel, Hq, Hkv, D, window, same = case
    q, kr, vr, kc, vc, sel, sinks = make_case(1, Sq, Sr, Sc, n_sel, Hq, Hkv, D, dtype, 1801)
    if same:
        vr, vc = kr, kc
    dev = lambda t: t.to(DEV)  # noqa: E731
    krd, kcd = dev(kr), dev(kc)
    vrd, vcd = (krd, kcd) if same else (dev(vr), dev(vc))
    for with_sinks in (True, False):
        s = sinks if with_sinks else None
        lse = torch.full((1, Hq, Sq), float("nan"), device=DEV)
        out = dtattn.sparse_indexed_attention(dev(q), krd, vrd, kcd, vcd, dev(sel) if n_sel else None, D ** -0.5,
                                              None if s is None else dev(s), window, lse=lse)
        torch.cuda.synchronize()
        ref, ref_lse = so.sparse_indexed_explicit(q, kr, vr, kc if n_sel else None, vc if n_sel else None, sel if n_sel else None,
                                                  D ** -0.5, s, window, compute_dtype=torch.float64, return_lse=True)
        mx, mean = so.error_stats(out.float().cpu(), ref.float())
        assert mx <= so.TOL_MAX_ABS + 2 * ROUND[dtype] * float(ref.abs().max()), (case, mx)
        assert mean <= so.TOL_MEAN_ABS + ROUND[dtype] * float(ref.abs().mean()), (case, mean)
        assert (lse.cpu().double() - ref_lse).abs().max() < 2e-3
