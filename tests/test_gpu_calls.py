"""The Python surface's calls in native code: what they serve, what they leave to the Python path, and that both answer alike."""
import pytest
import torch

from test_gpu_masked_prefill import make_mask
from test_gpu_parity import DEV, inputs

pytestmark = pytest.mark.gpu


@pytest.fixture
def python_only(dtattn, monkeypatch):
    """Switches the native calls off."""
    def off():
        class Declines:
            def __getattr__(self, name):
                return lambda *a: None
        monkeypatch.setattr(dtattn, "_calls", Declines())
    return off


def bits(t):
    return [x.clone().view(torch.int16 if x.element_size() == 2 else torch.int32) for x in (t if isinstance(t, (tuple, list)) else [t])]


def test_both_paths_answer_alike(dtattn, python_only):
    H = torch.float16
    q, k, v = (x.to(DEV) for x in inputs(2, 200, 300, 8, 4, 64, H, 2001))
    mask, sinks = make_mask(1, 1, 200, 300, H, 2002).to(DEV), torch.randn(8, device=DEV).to(H)
    odd = torch.zeros(200 * 301, device=DEV, dtype=H).view(1, 1, 200, 301)[..., 1:].copy_(mask)
    qd = q[:, :1]
    f = [x.float() for x in (q, k, v)]
    kc, vc = torch.zeros(1, 400, 2, 128, device=DEV, dtype=H), torch.zeros(1, 400, 2, 128, device=DEV, dtype=H)
    qs, kn, vn = (x.to(DEV) for x in inputs(1, 1, 1, 8, 2, 128, H, 2003))
    w, rot = torch.randn(128, device=DEV).to(H), torch.randn(1, 1, 128, device=DEV).to(H)
    px, pr = torch.randn(1, 70, 4, 64, device=DEV).to(H), torch.randn(1, 70, 1, 64, device=DEV).to(H)
    sq, kr = torch.randn(1, 2, 64, 512, device=DEV).to(H), torch.randn(1, 90, 1, 512, device=DEV).to(H)
    sel = torch.randint(-1, 90, (1, 2, 33), device=DEV, dtype=torch.int32)
    si = torch.randn(64, device=DEV).to(H)
    lse = torch.zeros(2, 8, 200, device=DEV)
    cases = [
        lambda: dtattn.sdpa_forward(q, k, v, 0.125), lambda: dtattn.sdpa_forward(q, k, v, 0.125, True, lse=lse),
        lambda: dtattn.sdpa_forward(q, k, v, 0.125, mask=mask), lambda: dtattn.sdpa_forward(q, k, v, 0.125, mask=odd),
        lambda: dtattn.sdpa_forward(q, k, v, 0.125, True, sinks=sinks, sliding_window=70), lambda: dtattn.sdpa_forward(qd, k, v, 0.125),
        lambda: dtattn.sdpa_forward(q[..., :40], k[..., :40], v[..., :40], 0.2), lambda: dtattn.sdpa_forward(*f, 0.125),
        lambda: dtattn.sdpa_forward(q.transpose(1, 2).contiguous().transpose(1, 2), k, v, 0.125),
        lambda: dtattn.decode_step(qs, kc, vc, kn, vn, rot, 0.1, 399, q_norm_weight=w, k_norm_weight=w),
        lambda: dtattn.qk_prologue(px, px, q_weight=w[:64], k_weight=w[64:], rotary=pr, post_scale=0.5),
        lambda: dtattn.sparse_indexed_attention(sq, kr, kr, kr, kr, sel, 0.05, si, 16)]
    cases[5]()  # (the device's own workspace is there from now on)
    native = [bits(fn()) for fn in cases]
    kept = [kc.clone(), vc.clone(), lse.clone()]
    python_only()
    for a, fn in zip(native, cases):
        b = bits(fn())
        assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b))
    assert all(torch.equal(x, y) for x, y in zip(kept, (kc, vc, lse)))
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0


def test_what_is_left_to_the_python_path(dtattn):
    q, k, v = (x.to(DEV) for x in inputs(1, 64, 64, 2, 2, 64, torch.float16, 2011))
    sdpa = lambda *a: dtattn._calls.sdpa(*a, None, 0.125, False, None, None, 0, None, 0, 0, 0, 0)  # noqa: E731
    assert isinstance(sdpa(q, k, v), torch.Tensor)

    class Sub(torch.Tensor):
        pass

    for t in (q.as_subclass(Sub), q.cpu(), q[0], q.double(), q.transpose(2, 3), q.float(), None, 3):
        assert sdpa(t, k, v) is None and sdpa(q, t, v) is None
    seen = []
    torch.vmap(lambda x: (seen.append(sdpa(x, k, v)), x)[1])(q[None])
    assert seen == [None]
    for bad in (dict(scale="x"), dict(mask=q), dict(lse=torch.zeros(3, device=DEV)), dict(sinks=k[0, 0, :, 0].float())):
        with pytest.raises((AssertionError, TypeError, dtattn.DtError)):
            dtattn.sdpa_forward(q, k, v, **dict(dict(scale=0.125), **bad))
    with pytest.raises(TypeError):
        dtattn._calls.sdpa(q, k, v)
    out = torch.zeros_like(q)
    assert dtattn.sdpa_forward(q, k, v, 0.125, out=out) is out
    assert dtattn.sdpa_forward(q, k, v, 1).shape == q.shape  # (a whole number as the scale)


def test_what_a_dispatch_mode_raises(dtattn):
    """An exception from Python code that torch runs inside a native call arrives as it was raised."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Refuses(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            raise ValueError("refused")

    x, row = (torch.zeros(1, n, 2, 64, dtype=torch.float16, device=DEV) for n in (4, 1))
    for call in (lambda: dtattn.sdpa_forward(x, x, x, 0.125), lambda: dtattn.qk_prologue(x, x),
                 lambda: dtattn.decode_step(row, x, x, row, row, None, 0.125, 3),
                 lambda: dtattn.sparse_indexed_attention(x, x, x, None, None, None, 0.125)):
        call()
        with pytest.raises(ValueError, match="refused"), Refuses():
            call()


def test_both_paths_refuse_alike(dtattn, python_only):
    """The same exception with the same text, whichever path a call takes first.  (Every call here is refused on the host.)"""
    H = torch.float16
    q, k, v = (x.to(DEV) for x in inputs(1, 64, 64, 4, 2, 64, H, 2021))
    mask, lse, sinks = torch.zeros(1, 1, 64, 64, device=DEV, dtype=H), torch.zeros(1, 4, 64, device=DEV), torch.zeros(4, device=DEV, dtype=H)
    row, kn, rot, w = q[:, :1], k[:, :1].clone(), torch.zeros(1, 1, 64, device=DEV, dtype=H), torch.zeros(64, device=DEV, dtype=H)
    table, sel = torch.zeros(1, 64, 1, 64, device=DEV, dtype=H), torch.zeros(1, 64, 8, device=DEV, dtype=torch.int32)
    wide = torch.zeros(1, 4, 4, 1024, device=DEV, dtype=H)
    nan = float("nan")
    sdpa = lambda **kw: dtattn.sdpa_forward(**dict(dict(q=q, k=k, v=v, scale=0.125), **kw))  # noqa: E731
    step = lambda **kw: dtattn.decode_step(**dict(dict(q=row, k_cache=k, v_cache=v, k_new=kn, v_new=kn, rotary=rot, scale=0.125,  # noqa: E731
                                                       cached_len=63), **kw))
    prologue = lambda **kw: dtattn.qk_prologue(**dict(dict(q=q, k=k, q_weight=w, k_weight=w, rotary=table), **kw))  # noqa: E731
    sparse = lambda **kw: dtattn.sparse_indexed_attention(**dict(dict(q=q, k_raw=k, v_raw=v, k_comp=k, v_comp=v, selected=sel,  # noqa: E731
                                                                      scale=0.125), **kw))
    refused = [
        (sdpa, kw) for kw in (dict(q=q[0]), dict(q=q.transpose(2, 3)), dict(q=q.double(), k=k.double(), v=v.double()), dict(scale="x"), dict(scale=nan),
                              dict(sliding_window=-1), dict(mask=mask[0]), dict(mask=mask[..., :63]), dict(mask=mask.float()),
                              dict(mask=mask.transpose(2, 3)), dict(lse=lse[..., :63]), dict(lse=lse.to(H)), dict(sinks=sinks[:3]), dict(sinks=sinks.float()),
                              dict(q=q[:, :, :3]), dict(q=wide, k=wide, v=wide), dict(flags="x"), dict(sliding_window="x"))] + [
        (step, kw) for kw in (dict(cached_len=63.0), dict(cached_len="x"), dict(rotary=rot[0]), dict(rotary=rot.float()), dict(rotary=rot[:, :0]),
                              dict(q_norm_weight=w[:63]), dict(k_norm_weight=w.float()), dict(scale=nan), dict(sliding_window=-1),
                              dict(lse=lse), dict(sinks=sinks[:3]), dict(norm_eps="x"), dict(q=q))] + [
        (prologue, kw) for kw in (dict(q=q[0]), dict(q_weight=w[:63]), dict(k_weight=w.float()), dict(rotary=table[0]), dict(rotary=table[:, :63]),
                                  dict(rotary=table.float()), dict(rotary_k=table[..., :32]), dict(eps="x"), dict(norm_per_token=True),
                                  dict(q=q.double(), q_weight=None, rotary=None))] + [
        (sparse, kw) for kw in (dict(q=q[0]), dict(selected=sel.long()), dict(selected=sel[0]), dict(selected=sel[:, :63]), dict(scale=nan),
                                dict(sliding_window=-1), dict(sinks=sinks[:3]), dict(sinks=sinks.float()), dict(lse=lse[..., :63]), dict(lse=lse.to(H)),
                                dict(q=q[:, :, :3]), dict(q=wide, k_raw=wide, v_raw=wide, k_comp=None, v_comp=None, selected=None), dict(scale="x"))]

    def answers():
        out = []
        for call, kw in refused:
            with pytest.raises(Exception) as e:
                call(**kw)
            out.append((call, list(kw), e.type, str(e.value)))
        return out

    native = answers()
    python_only()
    for a, b in zip(native, answers()):
        assert a == b
    torch.cuda.synchronize()
    assert dtattn.device_status() == 0
