"""The CPython binding of the forward calls: what it refuses, and how it treats outputs, streams and names."""
import ctypes as C
import gc

import numpy as np
import pytest
import torch

from llm170_b200 import _lib, synth

pytestmark = pytest.mark.gpu
N, K = 64, 256


@pytest.fixture(scope="module")
def dec():
    from llm170_b200.w4a16_dec import W4a16Dec
    d = W4a16Dec(0)
    for i, nm in enumerate(("a", "b")):
        q, s = synth.make_linear(N, K, 128, seed=40 + i)
        d.upload_lin_g(nm, q, s, N, K, 128)
    d.upload_head((np.arange(N * K, dtype=np.uint16) % 97 + 0x3f00).reshape(N, K), N, K)
    d.set_moe(8, 2, 64, K, 32, 0, 8)
    yield d
    d.close()


def x_of(t, seed=1):
    return torch.from_numpy(synth.make_acts(t, K, seed=seed).view(np.float16).copy()).cuda()


def bad_inputs(t, dtype):
    good = torch.zeros((t, K), device="cuda", dtype=dtype)
    return {"size": good[:, : K - 8].contiguous(), "type": good.to(torch.float64), "strides": torch.zeros((K, t), device="cuda", dtype=dtype).T,
            "device": good.cpu()}


@pytest.mark.parametrize("what", ["size", "type", "strides", "device"])
@pytest.mark.parametrize("t", [2, 16])
def test_refused_inputs_and_outputs(dec, what, t):
    from llm170_b200.w4a16_dec import W4a16Error
    x, bx = x_of(t), bad_inputs(t, torch.float16)[what]
    x32, bx32 = x.float(), bad_inputs(t, torch.float32)[what]
    by = {"size": torch.empty((t, N + 1), device="cuda"), "type": torch.empty((t, N), device="cuda", dtype=torch.float16),
          "strides": torch.empty((N, t), device="cuda").T, "device": torch.empty((t, N))}[what]
    calls = [lambda x, y: dec.lin_forward("a", x, t, dst=y), lambda x, y: dec.sk_multi_dev(["b", "a"], x, [None, y], t=t)]
    if t <= 8:
        calls += [lambda x, y: dec.sk_single_dev("a", x, out=y, t=t), lambda x, y: dec.sk_single_static("a", x, out=y, t=t)]
    for call in calls:
        with pytest.raises(W4a16Error):
            call(bx, None)
        with pytest.raises(W4a16Error):
            call(x, by)
    for call in (lambda x, y: dec.lin_forward_x32("a", x, t, dst=y), lambda x, y: dec.head_forward(x, t, out=y)):
        with pytest.raises(W4a16Error):
            call(bx32, None)
        with pytest.raises(W4a16Error):
            call(x32, by)
    logits = torch.zeros((t, 8), device="cuda")
    with pytest.raises(W4a16Error):
        dec.moe_ffn_dev_t(0, logits, bx, t)
    with pytest.raises(W4a16Error):
        dec.moe_ffn_dev_t(0, logits[:, :7].contiguous() if what == "size" else logits.double(), x, t)


def test_refused_names_lists_and_decoders(dec):
    from llm170_b200.w4a16_dec import W4a16Dec, W4a16Error
    x = x_of(1)
    for call in (lambda: dec.lin_forward("nowhere", x, 1), lambda: dec.sk_multi_dev(["a", "nowhere"], x),
                 lambda: dec.sk_multi_dev([], x), lambda: dec.sk_multi_dev(["a", "b"], x, [None])):
        with pytest.raises(W4a16Error):
            call()
    extra = torch.full((1, N), 7.0, device="cuda")
    assert len(dec.sk_multi_dev(["a", "b"], x, [None, None, extra])) == 2       # as zip() pairs them up
    dec.sync()
    assert bool((extra == 7.0).all())
    d = W4a16Dec(0)
    d.close()
    with pytest.raises(W4a16Error):
        d.lin_forward("a", x, 1)


def test_outputs_are_the_callers_or_come_from_torch(dec):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.ops = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.ops.append(str(func))
            return func(*args, **(kwargs or {}))

    x = x_of(3)
    dst = torch.empty((3, N), device="cuda")
    assert dec.lin_forward("a", x, 3, dst=dst) is dst
    with Seen() as seen:
        y = dec.lin_forward("a", x, 3)
    assert any("empty" in op for op in seen.ops), seen.ops       # what watches torch's allocations sees these too
    dec.sync()
    assert torch.equal(y, dst) and y.shape == (3, N) and y.dtype == torch.float32


@pytest.mark.parametrize("t", [1, 16])
def test_calls_run_on_torchs_current_stream(dec, t):
    x, new = x_of(t), x_of(t, seed=2)
    want = dec.lin_forward("a", new, t)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)        # x is still the old one when the call is made
        x.copy_(new)
        y = dec.lin_forward("a", x, t)
    side.synchronize()
    assert torch.equal(y, want)


class library_call:
    """One entry point of the library replaced by a host function."""

    def __init__(self, symbol, stand_in):
        self.symbol, self.stand_in = symbol, stand_in

    def _bind(self, stand_in):
        from llm170_b200.w4a16_dec import W4a16Error
        L = _lib.lib()
        own = lambda s: C.cast(getattr(L, s), C.c_void_p).value  # noqa: E731
        at = lambda s: C.cast(stand_in, C.c_void_p).value if stand_in and s == self.symbol else own(s)  # noqa: E731
        _lib.native(W4a16Error).bind(W4a16Error, at)

    def __enter__(self):
        self._bind(self.stand_in)

    def __exit__(self, *_):
        self._bind(None)


def test_new_outputs_are_filled_in_deterministic_mode(dec):
    x = x_of(2)

    @C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_char_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p)
    def writes_nothing(*_):
        return 0

    torch.use_deterministic_algorithms(True)
    try:
        with library_call("w4a16_lin_forward", writes_nothing):
            y = dec.lin_forward("a", x, 2)
    finally:
        torch.use_deterministic_algorithms(False)
    assert bool(torch.isnan(y).all())


def test_names_outlive_the_callers_list(dec):
    # the library runs without the interpreter lock: another thread may change the list of names meanwhile
    seen = []
    names = ["".join(["lin", str(i)]) for i in (900, 901)]
    for nm in names:
        q, s = synth.make_linear(N, K, 128, seed=44)
        dec.upload_lin_g(nm, q, s, N, K, 128)
    want = [nm.encode() for nm in names]
    del nm

    @C.CFUNCTYPE(C.c_int, C.c_void_p, C.POINTER(C.c_char_p), C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p)
    def in_the_library(_dec, nm, ns, _x, _outs, _t, _kind, _stream):
        names.clear()
        gc.collect()
        keep = [("other%d" % i) for i in range(64)]      # takes the place of freed strings
        seen.extend(nm[i] for i in range(ns))
        return len(keep) - 64

    x = x_of(1)
    with library_call("w4a16_sk_multi_dev", in_the_library):
        dec.sk_multi_dev(names, x)
    assert seen == want
