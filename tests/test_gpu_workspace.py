"""One workspace serves calls of different kinds one after another: each leaves what the next one relies on."""
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
