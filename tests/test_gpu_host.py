"""The native host path (csrc/host.cpp) against the Python bodies of the same functions: the same bits where it answers, and
no answer where the Python body has to decide."""
import pytest
import torch

pytestmark = pytest.mark.gpu
E4M3 = torch.float8_e4m3fn
BF16 = torch.bfloat16


class _NoHost:
    """Stands in for the extension: answers nothing, so the Python body runs."""

    def __getattr__(self, name):
        return lambda *a: None


class _Counting:
    def __init__(self, host):
        self.host, self.answers = host, []

    def __getattr__(self, name):
        def call(*a):
            r = getattr(self.host, name)(*a)
            self.answers.append((name, r is not None))
            return r
        return call


def _cases(dev):
    g = torch.Generator(device=dev).manual_seed(7)

    def r(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    def i8(*shape):
        return torch.randint(-127, 128, shape, generator=g, device=dev, dtype=torch.int8)
    x, cos, sin = r(2, 33, 512).to(BF16), r(1, 33, 512), r(1, 33, 512)
    sa, sb, bias = r(66).abs(), r(96).abs(), r(96)
    qkv = r(2, 33, 1536).to(BF16)
    heads = r(2, 33, 8, 64).to(BF16).transpose(1, 2)
    h8 = [r(2, 8, n, 64).to(E4M3) for n in (33, 70, 70)]
    lens = torch.tensor([70, 3], dtype=torch.int32, device=dev)
    row = (r(2, 1, 512).to(BF16), r(2, 1, 512).to(BF16))
    w8 = i8(96, 512)
    return {
        "tokenwise_quant": [(x, None), (x, E4M3)],
        "hadamard_quant": [(x, 0.05, None), (x.to(E4M3), 0.05, E4M3)],
        "fast_hadamard_transform": [(x, 0.05, None), (x, 0.05, E4M3)],
        "norm_modulate_quant": [(x,) + row + (None,)],
        "transpose_quant": [(w8, sb), (x[0, :32].contiguous(), None)],
        "dequant_hadamard": [(w8, sb, 0.05)],
        "rms_norm": [(x, None, None), (x, r(512), BF16)],
        "rms_norm_backward": [(x, sa.view(2, 33), x, r(512), None)],
        "rope": [(x, cos, sin, None), (x, cos.expand(2, -1, -1).contiguous(), sin.expand(2, -1, -1).contiguous(), torch.float32)],
        "rope_backward": [(x, cos, sin, BF16)],
        "q8_mm_bias": [(i8(2, 33, 512), w8, bias, sa, sb, True, BF16)],
        "q8_mm": [(i8(2, 33, 512), w8, sa, sb, False, None)],
        "fp8_mm": [(x.to(E4M3), w8.to(BF16).to(E4M3), sa, sb, False, BF16)],
        "mm_gate_residual": [(i8(2, 33, 512), w8, bias, sa, sb, r(2, 1, 96).to(BF16), r(2, 33, 96).to(BF16)),
                             (i8(2, 33, 512), w8, None, sa, sb, None, r(2, 33, 96).to(BF16))],
        "linear": [(x, w8, sb, bias, True, True, BF16), (x[0], w8.to(BF16).to(E4M3), sb, None, False, False, BF16)],
        "flash_attention": [(*h8, 0.125, None, None, False, True), (*h8, 0.125, lens, BF16, True, True)],
        "attention_prep_rows": [(heads, heads, heads, True, 0.05)],
        "qk_norm_rope_prep": [(qkv[..., :512], r(512), (cos, sin), 8, True, 0.05), (qkv[..., :512], r(512), None, 8, False, 1.0)],
        "kv_prep": [(qkv[..., :512], qkv[..., 512:1024], r(512), 8, True, 0.05)],
        "qk_norm_rope_prep_pair": [(qkv[..., :512], qkv[..., 512:1024], r(512), r(512), (cos, sin), 8, True, 0.05),
                                   (qkv[..., :512], qkv[..., 512:1024], r(512), r(512), None, 8, True, 0.05, qkv[..., 1024:])],
    }


def _flat(r):
    return [r] if isinstance(r, torch.Tensor) else list(r)


def _bits(t):
    return t.contiguous().view({1: torch.uint8, 2: torch.int16, 4: torch.int32}[t.element_size()])


def test_host_path_gives_what_the_python_bodies_give(cuda_device, monkeypatch):
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    host = native._host
    for name, calls in _cases(cuda_device).items():
        for args in calls:
            counting = _Counting(host)
            monkeypatch.setattr(native, "_host", counting)
            got = getattr(native, name)(*args)
            assert counting.answers and counting.answers[0][1], f"{name}: the native path did not answer"
            monkeypatch.setattr(native, "_host", _NoHost())
            want = getattr(native, name)(*args)
            assert type(got) is type(want), name
            for a, b in zip(_flat(got), _flat(want)):
                assert a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype, name
                assert torch.equal(_bits(a), _bits(b)), name


def test_host_path_leaves_everything_else_to_python(cuda_device):
    """Strided, wrapped, traced and mistyped arguments, and what is to be refused: None, and the Python body's own error."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from q8_kernels_b200 import _host, native

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    x = torch.randn(4, 32, 512, device=cuda_device).to(BF16)
    assert _host.hadamard_quant(x, 0.05, None) is not None
    assert _host.hadamard_quant(x[:, ::2], 0.05, None) is None
    assert _host.hadamard_quant(x.cpu(), 0.05, None) is None
    assert _host.hadamard_quant(x, 1, None) is None              # not a float
    assert _host.hadamard_quant(x, 0.05) is None
    assert _host.hadamard_quant(x, 0.05, BF16) is None
    with Mode():
        assert _host.hadamard_quant(x, 0.05, None) is None
    assert torch.func.vmap(lambda t: torch.tensor(_host.hadamard_quant(t, 0.05, None) is None))(x).all()
    with pytest.raises(native.Q8KernelError):
        native.hadamard_quant(x, 0.05, BF16)
    with pytest.raises(native.Q8KernelError):                   # refused by the kernel's entry point, not by a check before it
        native.fast_hadamard_transform(torch.zeros(2, 32768, device=cuda_device, dtype=BF16), 1.0)
    with pytest.raises(native.Q8KernelError):
        native.q8_mm(x.to(E4M3), x[0].to(E4M3), torch.ones(128, device=cuda_device), torch.ones(32, device=cuda_device), False, BF16)


def test_pre_passes_refuse_what_their_python_bodies_refuse(cuda_device, monkeypatch):
    """None in a required place, in the rotary tables too, is no shorter form of the call; other sequences of the two tables are
    taken as before."""
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    qkv = torch.randn(2, 33, 1536, device=cuda_device).to(BF16)
    q, k, v = qkv[..., :512], qkv[..., 512:1024], qkv[..., 1024:]
    w = torch.rand(512, device=cuda_device)
    cos, sin = torch.randn(1, 33, 512, device=cuda_device), torch.randn(1, 33, 512, device=cuda_device)
    refused = [(native.kv_prep, (k, None, w, 8, True, 0.05)), (native.kv_prep, (None, v, w, 8, True, 0.05)),
               (native.kv_prep, (k, v, None, 8, True, 0.05)), (native.qk_norm_rope_prep, (q, None, None, 8, True, 0.05)),
               (native.qk_norm_rope_prep, (q, w, (None, None), 8, True, 0.05)), (native.qk_norm_rope_prep, (q, w, (cos,), 8, True, 0.05)),
               (native.qk_norm_rope_prep, (q, w, (cos, sin, cos), 8, True, 0.05)), (native.qk_norm_rope_prep, (q, w, None, 2 ** 58 + 8, True, 0.05)),
               (native.qk_norm_rope_prep_pair, (None, k, None, w, None, 8, True, 0.05)),
               (native.qk_norm_rope_prep_pair, (None, k, None, w, None, 8, True, 0.05, v)),
               (native.qk_norm_rope_prep_pair, (q, k, None, w, None, 8, True, 0.05)),
               (native.qk_norm_rope_prep_pair, (q, k, w, w, (cos, None), 8, True, 0.05))]
    for fn, args in refused:
        with pytest.raises((AttributeError, ValueError, native.Q8KernelError)):
            fn(*args)
    with monkeypatch.context() as m:
        m.setattr(native, "_host", _NoHost())
        want = native.qk_norm_rope_prep(q, w, (cos, sin), 8, True, 0.05)
    for freqs in ((cos, sin), [cos, sin], iter((cos, sin)), torch.stack((cos, sin))):
        assert torch.equal(_bits(native.qk_norm_rope_prep(q, w, freqs, 8, True, 0.05)), _bits(want))


def test_an_error_of_a_product_names_the_function_that_was_called(cuda_device):
    from q8_kernels_b200 import native
    a = torch.ones(4, 24, dtype=torch.int8, device=cuda_device)  # K is no multiple of 16
    s, bias = torch.ones(4, device=cuda_device), torch.zeros(4, device=cuda_device)
    f = torch.ones(4, 24, device=cuda_device).to(E4M3)
    for name, call in (("q8_mm", lambda: native.q8_mm(a, a, s, s, False)), ("q8_mm_bias", lambda: native.q8_mm_bias(a, a, bias, s, s, False)),
                       ("fp8_mm", lambda: native.fp8_mm(f, f, s, s, False)), ("fp8_mm_bias", lambda: native.fp8_mm_bias(f, f, bias, s, s, False))):
        with pytest.raises(native.Q8KernelError, match=f"^{name}: "):
            call()


def test_a_linear_holds_no_scratch_after_the_call(cuda_device, monkeypatch):
    """Neither path keeps memory: what is allocated after a call is its result."""
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    x = torch.randn(2, 1000, 512, device=cuda_device).to(BF16)[:, ::2]          # strided: the Python body's
    w = torch.ones(96, 512, dtype=torch.int8, device=cuda_device)
    s = torch.ones(96, device=cuda_device)
    for t in (x, x.contiguous()):
        for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                held = torch.cuda.memory_allocated()
                out = native.linear(t, w, s, None, True, False, BF16)
                assert torch.cuda.memory_allocated() - held == (out.nbytes + 511) // 512 * 512
                del out
    torch.cuda.synchronize()


class _Recording(_Counting):
    def __getattr__(self, name):
        def call(*a):
            r = getattr(self.host, name)(*a)
            self.answers.append((name, a, r))
            return r
        return call


# places of the extension's functions that may be None
_OPTIONAL = {("transpose_quant", 1), ("rms_norm", 1), ("rms_norm_backward", 3), ("mm", 2), ("mm_gate_residual", 2), ("mm_gate_residual", 5),
             ("linear", 3), ("flash_attention", 4), ("qk_norm_rope_prep_pair", 8)}


def test_host_path_takes_nothing_else_in_the_place_of_a_tensor(cuda_device, monkeypatch):
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    host = native._host
    for name, calls in _cases(cuda_device).items():
        for args in calls:
            recording = _Recording(host)
            with monkeypatch.context() as m:
                m.setattr(native, "_host", recording)
                getattr(native, name)(*args)
            fn, a, answer = recording.answers[0]
            assert answer is not None
            for i, t in enumerate(a):
                if isinstance(t, torch.Tensor):
                    for other in (3, t.cpu(), t.double()) + (() if (fn, i) in _OPTIONAL else (None,)):
                        assert getattr(host, fn)(*a[:i], other, *a[i + 1:]) is None, (fn, i, type(other))


def _map(args, f):
    return tuple(f(a) if isinstance(a, torch.Tensor) else tuple(map(f, a)) if isinstance(a, tuple) else a for a in args)


def _same(got, want, name):
    for a, b in zip(_flat(got), _flat(want)):
        assert torch.equal(_bits(a), _bits(b)), name


def test_host_path_launches_on_the_current_stream(cuda_device):
    """Inputs that another stream fills late, behind a delay: only work queued on that stream sees them."""
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    side = torch.cuda.Stream()
    for name, calls in _cases(cuda_device).items():
        for args in calls:
            want = getattr(native, name)(*args)
            late = _map(args, torch.zeros_like)
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                torch.cuda._sleep(1_000_000)
                for to, t in zip(late, args):
                    for x, y in zip(to, t) if isinstance(t, tuple) else [(to, t)] if isinstance(t, torch.Tensor) else []:
                        x.copy_(y)
                got = getattr(native, name)(*late)
            side.synchronize()
            _same(got, want, name)


def test_host_path_under_capture(cuda_device):
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    for name, calls in _cases(cuda_device).items():
        for args in calls:
            want = getattr(native, name)(*args)
            static = _map(args, torch.zeros_like)
            getattr(native, name)(*static)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                got = getattr(native, name)(*static)
            for to, t in zip(static, args):
                for x, y in zip(to, t) if isinstance(t, tuple) else [(to, t)] if isinstance(t, torch.Tensor) else []:
                    x.copy_(y)
            graph.replay()
            torch.cuda.synchronize()
            _same(got, want, name)


def test_host_path_from_several_threads(cuda_device):
    """The interpreter lock is given up inside a call: threads on streams of their own, all functions at once."""
    import threading
    from q8_kernels_b200 import _lib, native
    _lib.status_word(cuda_device)
    calls = [(name, args, getattr(native, name)(*args)) for name, c in _cases(cuda_device).items() for args in c]
    torch.cuda.synchronize()
    failed = []

    def work(first):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(3 * len(calls)):
                    name, args, want = calls[(first + i) % len(calls)]
                    _same(getattr(native, name)(*args), want, name)
        except BaseException as e:                              # (an assertion too: it must reach the test)
            failed.append(e)
    threads = [threading.Thread(target=work, args=(k * 5,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
