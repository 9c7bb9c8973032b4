"""Scratch: one workspace serves calls of different kinds one after another, and each leaves what the next one relies on; the
scratch of a call belongs to the stream that the call runs on."""
import pytest
import torch

from test_gpu_masked_prefill import make_mask
from test_gpu_parity import DEV, inputs

pytestmark = pytest.mark.gpu


def test_masked_calls_leave_the_ticket_counters_alone(dtattn):
    """A masked prompt and a decode step through the same workspace: the split-KV tickets in its first 4 KB stay zero."""
    q, k, v = (x.to(DEV) for x in inputs(1, 512, 512, 8, 8, 64, torch.float16, 1421))
    mask = make_mask(1, 1, 512, 512, torch.float16, 1422).to(DEV)
    ws = dtattn.Workspace(torch.device(DEV))
    dq, dk, dv = (x.to(DEV) for x in inputs(1, 1, 8192, 32, 8, 128, torch.float16, 1423))
    want = dtattn.sdpa_forward(dq, dk, dv, 128 ** -0.5, workspace=ws)
    dtattn.sdpa_forward(q, k, v, 0.125, mask=mask, workspace=ws)
    got = dtattn.sdpa_forward(dq, dk, dv, 128 ** -0.5, workspace=ws, out=torch.zeros_like(dq))
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("kind", ["cut", "fp32", "unaligned mask"])
def test_scratch_is_in_the_order_of_the_calls_stream(dtattn, kind):
    """A call with stream=, while the current stream still has kernels queued that write to a block torch has already taken
    back: the call's scratch is not that block."""
    dtype = torch.float32 if kind == "fp32" else torch.bfloat16
    Sq, Sk = (200, 4096) if kind == "cut" else (333, 333)
    q, k, v = (x.to(DEV) for x in inputs(1, Sq, Sk, 4, 4, 64, dtype, 1431))
    mask = make_mask(1, 1, Sq, Sk, dtype, 1432).to(DEV) if kind == "unaligned mask" else None
    want = dtattn.sdpa_forward(q, k, v, 0.125, mask=mask)
    out, side = torch.zeros_like(want), torch.cuda.Stream()
    need = dtattn.workspace_size(dtattn.make_params(q, k, v, out, 0.125, mask=mask))
    assert need > 0
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # the only free block of this size is the one below
    for _ in range(3):
        busy = torch.empty(need, dtype=torch.uint8, device=DEV)
        torch.cuda._sleep(int(2e6))  # a millisecond or so, while the rest is queued
        for _ in range(400):
            busy.fill_(0x7f)
        del busy
        for _ in range(60):  # over the sleep and into the fills
            dtattn.sdpa_forward(q, k, v, 0.125, mask=mask, out=out, stream=side.cuda_stream)
        torch.cuda.synchronize()
        assert dtattn.device_status() == 0
        assert torch.equal(out, want)
        out.zero_()
        torch.cuda.synchronize()


@pytest.mark.parametrize("kind", ["cut", "fp32", "unaligned mask", "aligned mask", "decode"])
@pytest.mark.parametrize("own", [False, True])
def test_no_room_for_scratch(dtattn, monkeypatch, kind, own):
    """Scratch that only makes a call faster may be missing, with a caller's workspace as without; what a call cannot do
    without is torch's out-of-memory error."""
    dtype = torch.float32 if kind == "fp32" else torch.bfloat16
    Sq, Sk = {"cut": (200, 4096), "decode": (1, 4096), "aligned mask": (512, 512)}.get(kind, (333, 333))
    q, k, v = (x.to(DEV) for x in inputs(1, Sq, Sk, 4, 4, 64, dtype, 1441))
    mask = make_mask(1, 1, Sq, Sk, dtype, 1442).to(DEV) if kind.endswith("mask") else None
    want = dtattn.sdpa_forward(q, k, v, 0.125, mask=mask)
    torch.cuda.synchronize()

    def no_room(nbytes, device, stream):
        raise torch.cuda.OutOfMemoryError("no room")

    monkeypatch.setattr(dtattn, "_alloc", no_room)
    monkeypatch.setattr(dtattn, "_workspaces", {})
    kw = dict(workspace=dtattn.Workspace(torch.device(DEV))) if own else {}
    if kind in ("aligned mask", "decode"):
        with pytest.raises(torch.cuda.OutOfMemoryError):
            dtattn.sdpa_forward(q, k, v, 0.125, mask=mask, **kw)
        return
    got = dtattn.sdpa_forward(q, k, v, 0.125, mask=mask, **kw)
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    assert float((got.float() - want.float()).abs().max()) <= (4e-5 if kind == "fp32" else 2 ** -7)


@pytest.mark.parametrize("Sk", [512, 4096])  # not cut; cut
def test_projected_calls_on_two_streams(dtattn, Sk):
    """The attention output of a projected call lives in scratch: calls on several streams keep theirs apart."""
    H, D, dtype = 4, 64, torch.float16
    cases, streams = [], [torch.cuda.Stream(), torch.cuda.Stream()]
    for i in range(2):
        q, k, v = (x.to(DEV) for x in inputs(1, 256, Sk, H, H, D, dtype, 1451 + 10 * i))
        w = (torch.randn(H * D, H * D, generator=torch.Generator().manual_seed(i)) / 16).to(dtype).to(DEV)
        cases.append((q, k, v, 0.125, w))
    wants = [dtattn.sdpa_forward_projected(*c) for c in cases]
    torch.cuda.synchronize()
    outs = [[], []]
    for _ in range(40):
        for i, c in enumerate(cases):
            with torch.cuda.stream(streams[i]):
                outs[i].append(dtattn.sdpa_forward_projected(*c))
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
    for i in range(2):
        assert all(torch.equal(o, wants[i]) for o in outs[i])
