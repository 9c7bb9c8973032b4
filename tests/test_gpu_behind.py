"""Launches whose CTAs may start while the kernel before them runs out: results do not depend on it.  Every call here reads what the one
before it wrote, or overwrites what the one before it reads, on one stream without a synchronisation, against the same calls one
at a time."""
import pytest
import torch

from test_gpu_masked_prefill import make_mask
from test_gpu_parity import DEV, inputs

pytestmark = pytest.mark.gpu


def chain(dtattn, s, wait):
    """One round over buffers that the calls hand from one to the next."""
    D = 64
    for i in range(3):
        s["x"].mul_(0.5).add_(s["y"], alpha=0.5)
        wait()
        dtattn.qk_prologue(s["x"], s["y"], q_out=s["q"], k_out=s["k"], q_weight=s["w"], k_weight=s["w"], rotary=s["rot"])
        wait()
        dtattn.sdpa_forward(s["q"], s["k"], s["x"], D ** -0.5, True, out=s["o"])
        wait()
        dtattn.sdpa_forward(s["o"], s["k"][:, :77], s["x"][:, :77], D ** -0.5, out=s["y"])  # short keys
        wait()
        dtattn.sdpa_forward(s["y"], s["k"], s["o"], D ** -0.5, mask=s["mask"], out=s["q"])  # a mask of odd rows: three kernels
        wait()
        dtattn.decode_step(s["q"][:, :1], s["kc"], s["vc"], s["k"][:, :1], s["o"][:, :1], s["rot"][:, :1, 0], D ** -0.5, 700 + i, out=s["d"])
        wait()
        s["x"][:, :1] = s["d"]
        wait()
        s["f"].copy_(s["x"])
        dtattn.sdpa_forward(s["f"], s["f"], s["f"], D ** -0.5, out=s["g"])
        wait()
        s["y"].copy_(s["g"])
        wait()
        s["y"] += dtattn.sdpa_forward_projected(s["q"], s["k"], s["o"], D ** -0.5, s["pw"]).view_as(s["y"])
        wait()


def buffers():
    H, D, S, dt = 4, 64, 333, torch.float16
    x, y, o = (t.to(DEV) for t in inputs(1, S, S, H, H, D, dt, 2101))
    s = dict(x=x, y=y, o=o, q=torch.empty_like(x), k=torch.empty_like(x), d=torch.empty_like(x[:, :1]), f=x.float(), g=x.float())
    s["kc"], s["vc"], _ = (t.to(DEV) for t in inputs(1, 1000, 1000, H, H, D, dt, 2102))
    s["mask"] = make_mask(1, 1, S, S, dt, 2103).to(DEV)
    g = torch.Generator().manual_seed(2104)
    s["w"] = torch.randn(D, generator=g).to(dt).to(DEV)
    s["rot"] = torch.randn(1, S, 1, D, generator=g).to(dt).to(DEV)
    s["pw"] = (torch.randn(H * D, H * D, generator=g) / 16).to(dt).to(DEV)
    return s


def test_a_chain_of_calls(dtattn):
    one = buffers()
    for _ in range(5):
        chain(dtattn, one, torch.cuda.synchronize)
    many = buffers()
    for _ in range(5):
        chain(dtattn, many, lambda: None)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    # in a graph, behind a copy, a memset and work of another stream
    graphed, side = buffers(), torch.cuda.Stream()
    keep = {k: v.clone() for k, v in graphed.items()}
    chain(dtattn, graphed, lambda: None)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        here = torch.cuda.current_stream()
        graphed["g"].zero_()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            graphed["d"].zero_()
        here.wait_stream(side)
        chain(dtattn, graphed, lambda: None)
    for k, v in keep.items():
        graphed[k].copy_(v)
    for _ in range(5):
        g.replay()
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    for k in one:
        assert torch.equal(one[k], many[k]) and torch.equal(one[k], graphed[k]), k


def test_a_stable_prefix_is_stable_behind_an_overlapped_call(dtattn):
    """The cache is written by a long copy, a small call of ours follows, and then a decode call that may stream its prefix while
    that small call runs: not while the copy does."""
    B, T, H, D, dt = 16, 4096, 8, 128, torch.bfloat16
    q, k, v = (t.to(DEV) for t in inputs(B, 1, T, H, H, D, dt, 2111))
    sq, sk, sv = (t.to(DEV) for t in inputs(1, 200, 77, 2, 2, 64, dt, 2112))
    kc, vc = torch.zeros_like(k), torch.zeros_like(v)
    want = dtattn.sdpa_forward(q, k, v, D ** -0.5, True)
    for _ in range(20):
        kc.zero_(), vc.zero_()
        kc.copy_(k), vc.copy_(v)
        dtattn.sdpa_forward(sq, sk, sv, 0.125)
        got = dtattn.sdpa_forward(q, kc, vc, D ** -0.5, True, flags=dtattn.DT_FLAG_KV_PREFIX_STABLE)
        assert torch.equal(got, want)
    assert dtattn.device_status() == 0
