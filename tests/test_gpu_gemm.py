"""GPU parity of the tcgen05 INT8 / FP8 GEMM against the CPU oracle (rel.
Frobenius <= 2e-3 on the bf16 output; the oracle is rounded to bf16 too), plus
size-independent properties at the full DiT shapes."""
import pytest
import torch

import golden_io as G
import helpers as Hp
from oracle import q8_oracle as O

pytestmark = pytest.mark.gpu
E4M3 = torch.float8_e4m3fn
TOL = 2e-3


@pytest.fixture(scope="module")
def nat(cuda_device):
    from q8_kernels_b200 import native
    return native


def _operands(M, N, K, kind, seed):
    a = Hp.activations(M, K, seed)
    w = Hp.weights(N, K, seed + 1)
    qd = torch.int8 if kind == "int8" else E4M3
    aq, sa = O.tokenwise_quant(a, qd)
    wq, sw = O.tokenwise_quant(w, qd)
    return aq, sa, wq, sw, Hp.bias_vec(N, seed + 2)


def _run(nat, dev, kind, aq, sa, wq, sw, bias, gelu, out_dtype):
    mm = {"int8": (nat.q8_mm, nat.q8_mm_bias), "fp8": (nat.fp8_mm, nat.fp8_mm_bias)}[kind]
    args = [t.to(dev) for t in (aq, wq)]
    if bias is not None:
        return mm[1](args[0], args[1], bias.to(dev), sa.to(dev), sw.to(dev), gelu, out_dtype)
    return mm[0](args[0], args[1], sa.to(dev), sw.to(dev), gelu, out_dtype)


def _oracle(kind, aq, sa, wq, sw, bias, gelu, out_dtype):
    f = O.q8_mm if kind == "int8" else O.fp8_mm
    return f(aq, wq, sa, sw, gelu, out_dtype, bias=bias)


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (128, 128, 128), (256, 512, 512), (100, 256, 256),
                                   (1, 128, 64), (300, 384, 192), (129, 640, 1024), (512, 2048, 2048),
                                   (77, 48, 80)])
def test_gemm_small_shapes(nat, cuda_device, kind, M, N, K):
    aq, sa, wq, sw, bias = _operands(M, N, K, kind, seed=M + N + K)
    got = _run(nat, cuda_device, kind, aq, sa, wq, sw, bias, False, torch.bfloat16)
    ref = _oracle(kind, aq, sa, wq, sw, bias, False, torch.bfloat16)
    assert got.shape == (1, M, N) and got.dtype == torch.bfloat16
    err = Hp.rel_fro(got.float(), ref.float())
    assert err <= TOL, f"rel fro {err:.3e}"
    if kind == "int8":
        # integer accumulation is exact, the epilogue differs from the oracle by at most an fma rounding
        flips = (Hp.bits(got.cpu()) != Hp.bits(ref)).float().mean().item()
        assert flips < 0.02, f"{flips:.4f} of bf16 outputs differ"


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("bias,gelu,out_dtype", [(False, False, torch.bfloat16), (True, True, torch.bfloat16),
                                                 (False, True, E4M3), (True, False, None)])
def test_gemm_epilogue_variants(nat, cuda_device, kind, bias, gelu, out_dtype):
    aq, sa, wq, sw, b = _operands(384, 512, 768, kind, seed=50)
    b = b if bias else None
    got = _run(nat, cuda_device, kind, aq, sa, wq, sw, b, gelu, out_dtype)
    ref = _oracle(kind, aq, sa, wq, sw, b, gelu, out_dtype)
    want_dtype = E4M3 if out_dtype in (None, E4M3) else out_dtype
    assert got.dtype == want_dtype                                   # default output dtype is e4m3, as in the reference
    if want_dtype == torch.bfloat16:
        assert Hp.rel_fro(got.float(), ref.float()) <= TOL
    else:
        # e4m3 output: compare as values; a 1-ulp flip is 6 %, so count flips instead of a norm
        g, r = got.float().cpu(), ref.float()
        assert not torch.isnan(g).any()
        flips = (g != r).float().mean().item()
        assert flips < 0.02, f"{flips:.4f} of e4m3 outputs differ"
        assert g.abs().max() <= 448


@pytest.mark.parametrize("kind", ["int8", "fp8"])
def test_gemm_batched_and_broadcast(nat, cuda_device, kind):
    qd = torch.int8 if kind == "int8" else E4M3
    a = Hp.activations(3 * 160, 256, seed=60).reshape(3, 160, 256)
    w = Hp.weights(3 * 128, 256, seed=61).reshape(3, 128, 256)
    aq, sa = O.tokenwise_quant(a, qd)
    wq, sw = O.tokenwise_quant(w, qd)
    f = nat.q8_mm if kind == "int8" else nat.fp8_mm
    d = cuda_device
    for (A, SA, W, SW) in [(aq, sa, wq, sw), (aq, sa, wq[0], sw[0]), (aq[1], sa[1], wq, sw)]:
        got = f(A.contiguous().to(d), W.contiguous().to(d), SA.contiguous().to(d), SW.contiguous().to(d), False,
                torch.bfloat16)
        ref = _oracle(kind, A, SA, W, SW, None, False, torch.bfloat16)
        assert got.shape == ref.shape == (3, 160, 128)
        assert Hp.rel_fro(got.float(), ref.float()) <= TOL


def test_gemm_golden_fixture(nat, cuda_device):
    d = G.load("oracle_gemm.npz")
    dev = cuda_device
    y = nat.q8_mm_bias(G.t(d["aq"]).to(dev), G.t(d["wq"]).to(dev), G.t(d["bias"]).to(dev), G.t(d["sa"]).to(dev),
                       G.t(d["sw"]).to(dev), True, torch.bfloat16)
    assert Hp.rel_fro(y.float(), G.bf16(d["y_i8"]).float()) <= TOL
    y = nat.fp8_mm_bias(G.e4m3(d["af"]).to(dev), G.e4m3(d["wf"]).to(dev), G.t(d["bias"]).to(dev),
                        G.t(d["saf"]).to(dev), G.t(d["swf"]).to(dev), True, torch.bfloat16)
    assert Hp.rel_fro(y.float(), G.bf16(d["y_f8"]).float()) <= TOL


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("K,N", [(2048, 2048), (2048, 6144), (2048, 8192), (8192, 2048)])
def test_gemm_full_dit_shapes_properties(nat, cuda_device, kind, K, N):
    """M = 6144 (one video).  The oracle is checked on a random sample of rows;
    the whole output is checked through linearity in the row scales (doubling
    sa doubles a bias-free output exactly) and a column-sum identity."""
    M = 6144
    aq, sa, wq, sw, bias = _operands(M, N, K, kind, seed=K + N)
    dev = cuda_device
    got = _run(nat, dev, kind, aq, sa, wq, sw, bias, True, torch.bfloat16)
    rows = torch.randperm(M, generator=Hp.gen(1))[:96]
    ref = _oracle(kind, aq[rows], sa[rows], wq, sw, bias, True, torch.bfloat16)
    err = Hp.rel_fro(got[0, rows.to(dev)].float(), ref[0].float())
    assert err <= TOL, f"rel fro {err:.3e}"
    plain = _run(nat, dev, kind, aq, sa, wq, sw, None, False, torch.bfloat16)
    doubled = _run(nat, dev, kind, aq, sa * 2, wq, sw, None, False, torch.bfloat16)
    assert torch.equal(doubled.float(), plain.float() * 2)              # exact: power-of-two scaling commutes with rounding
    # sum over rows of the fp32-exact product equals (sum of scaled A rows) . B^T
    a_deq = (aq.float() * sa[:, None]).to(torch.float64).sum(dim=0)
    col_ref = (wq.to(torch.float64) * sw[:, None].double()) @ a_deq
    col_got = plain[0].double().sum(dim=0).cpu()
    assert Hp.rel_fro(col_got, col_ref) < 5e-3                          # bf16 output rounding accumulates over 6144 rows


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("K,N", [(2048, 8192), (8192, 2048)])
def test_gemm_four_videos_of_tokens_sampled(nat, cuda_device, kind, K, N):
    """M = 24576 (four videos): sampled rows against the oracle, bias + tanh-GELU, bf16 out; plus exact
    power-of-two linearity of the whole bias-free output in the row scales."""
    M = 24576
    aq, sa, wq, sw, bias = _operands(M, N, K, kind, seed=3 * K + N)
    dev = cuda_device
    got = _run(nat, dev, kind, aq, sa, wq, sw, bias, True, torch.bfloat16)
    rows = torch.cat([torch.randperm(M, generator=Hp.gen(2))[:60], torch.tensor([0, 255, 256, M - 257, M - 1])])
    ref = _oracle(kind, aq[rows], sa[rows], wq, sw, bias, True, torch.bfloat16)
    err = Hp.rel_fro(got[0, rows.to(dev)].float(), ref[0].float())
    assert err <= TOL, f"rel fro {err:.3e}"
    plain = _run(nat, dev, kind, aq, sa, wq, sw, None, False, torch.bfloat16)
    halved = _run(nat, dev, kind, aq, sa * 0.5, wq, sw, None, False, torch.bfloat16)
    assert torch.equal(halved.float() * 2, plain.float())


def test_gemm_argument_errors(nat, cuda_device):
    from q8_kernels_b200._lib import Q8KernelError
    d = cuda_device
    a = torch.zeros(8, 64, dtype=torch.int8, device=d)
    w = torch.zeros(16, 64, dtype=torch.int8, device=d)
    sa = torch.ones(8, device=d)
    sw = torch.ones(16, device=d)
    with pytest.raises(Q8KernelError, match="contiguous"):
        nat.q8_mm(a.t().contiguous().t(), w, sa, sw, False, torch.bfloat16)
    with pytest.raises(Q8KernelError, match="K mismatch"):
        nat.q8_mm(a, torch.zeros(16, 32, dtype=torch.int8, device=d), sa, sw, False, torch.bfloat16)
    with pytest.raises(Q8KernelError):
        nat.fp8_mm(a, w, sa, sw, False, torch.bfloat16)                 # wrong operand dtype
    with pytest.raises(Q8KernelError, match="Batch missmatch"):
        nat.q8_mm(torch.zeros(2, 8, 64, dtype=torch.int8, device=d), torch.zeros(3, 16, 64, dtype=torch.int8, device=d),
                  torch.ones(2, 8, device=d), torch.ones(3, 16, device=d), False, torch.bfloat16)


def _check_epilogues(nat, d, kind, B, Bw, M, N, K):
    """Every epilogue against float64.  INT8 sums are exact and FP8 sums fp32, so a bf16 result is one rounding (at most
    2^-8 of the value: half of a step of 2^-7) and a few fp32 ones away; GELU adds half of |y| times the 2^-11 of
    tanh.approx; an e4m3 result is one rounding of 2^-4, or half of the subnormal step."""
    qd = torch.int8 if kind == "int8" else E4M3
    g = Hp.gen(M + N + K)

    def mk(*s):
        if kind == "int8":
            return torch.randint(-127, 128, s, generator=g, dtype=torch.int8).to(d)
        return torch.randn(s, generator=g).to(qd).to(d)

    ad, wd = mk(B, M, K), mk(*((Bw, N, K) if Bw > 1 else (N, K)))
    sad = (torch.rand(B, M, generator=g) * 0.01 + 0.001).to(d)
    swd = (torch.rand(*((Bw, N) if Bw > 1 else (N,)), generator=g) * 0.01 + 0.001).to(d)
    bd = (torch.randn(N, generator=g) * 0.1).to(d)
    y = (ad.double() @ wd.double().transpose(-1, -2)) * sad.double().unsqueeze(-1)
    y = y * (swd.double().unsqueeze(1) if Bw > 1 else swd.double()) + bd.double()
    fp32 = 2e-6 * y.abs().max()
    mm, mmb = (nat.q8_mm, nat.q8_mm_bias) if kind == "int8" else (nat.fp8_mm, nat.fp8_mm_bias)
    lin = mmb(ad, wd, bd, sad, swd, False, torch.bfloat16)
    assert bool(((lin.double() - y).abs() <= 2.0 ** -8 * y.abs() + fp32).all())
    ge = torch.nn.functional.gelu(y, approximate="tanh")
    out = mmb(ad, wd, bd, sad, swd, True, torch.bfloat16)
    assert bool(((out.double() - ge).abs() <= 2.0 ** -8 * ge.abs() + 1.02 * 2.0 ** -12 * y.abs() + fp32).all())
    out8 = mm(ad, wd, sad, swd, False, None)
    y8 = (y - bd.double()).clamp(-448, 448)
    assert bool(((out8.double() - y8).abs() <= 2.0 ** -3.9 * y8.abs() + 2.0 ** -9).all())
    if Bw == 1:
        gate = torch.randn(B, 1, N, generator=g).to(torch.bfloat16).to(d)
        resid = torch.randn(B, M, N, generator=g).to(torch.bfloat16).to(d)
        fused = nat.mm_gate_residual(ad, wd, bd, sad, swd, gate, resid)
        Hp.assert_bit_equal(fused, (gate * lin + resid).cpu(), "gate and residual in the epilogue")


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("B,M,N,K", [(1, 1, 16, 16), (1, 7, 48, 112), (2, 9, 2064, 640), (1, 77, 10240, 1040), (1, 127, 144, 4112),
                                     (1, 128, 2048, 2048), (3, 129, 272, 272), (1, 300, 2048, 2048), (1, 512, 2064, 8208),
                                     (2, 260, 1040, 1024), (1, 4000, 128, 512), (1, 1000, 96, 144)])
def test_split_tiles_and_split_k(nat, cuda_device, kind, B, M, N, K):
    """Shapes as they come: row / column / K tails and batches on shared weights, each epilogue."""
    _check_epilogues(nat, cuda_device, kind, B, 1, M, N, K)


@pytest.mark.parametrize("bn,sk,Bw,M,N,K", [
    (32, 1, 3, 33, 96, 272), (48, 1, 1, 120, 6160, 144), (64, 1, 2, 9, 4112, 272), (80, 1, 1, 400, 2576, 272),
    (96, 1, 1, 900, 1552, 272), (112, 1, 1, 260, 5136, 272), (128, 1, 2, 1000, 1040, 144), (144, 1, 3, 1000, 784, 144),
    (160, 1, 1, 1300, 2064, 144), (176, 1, 1, 511, 6160, 112), (208, 1, 1, 1300, 2576, 112), (224, 1, 3, 127, 10256, 112),
    (32, 2, 2, 77, 656, 4112), (48, 2, 1, 100, 3088, 4112), (64, 2, 3, 127, 1168, 4112), (80, 2, 3, 129, 784, 8208),
    (96, 2, 1, 127, 6160, 4112), (112, 2, 3, 129, 1168, 8208), (128, 2, 2, 129, 2064, 8208), (144, 2, 1, 129, 5136, 8208),
    (32, 4, 2, 100, 144, 4112), (64, 4, 2, 200, 528, 4112), (96, 4, 2, 260, 528, 8208), (96, 4, 1, 100, 3088, 8208)])
def test_every_tile_width_and_k_split(nat, cuda_device, bn, sk, Bw, M, N, K):
    """One shape per tile width and number of K shares that the dispatch uses on 148 SMs, with tails in every direction
    and, where there is one, a batch of weights.  The choice itself is asserted, so that another cost model cannot take the
    coverage away unnoticed.  FP8 takes the same width where K is not split, and never splits."""
    import ctypes
    from q8_kernels_b200 import _lib
    plan = (ctypes.c_int * 3)()
    for kind in ("int8", "fp8"):
        assert _lib.lib.q8k_mm_plan(int(kind == "int8"), Bw, Bw, M, N, K, ctypes.cast(plan, ctypes.c_void_p)) == 0
        assert tuple(plan) == (0, bn, sk) if kind == "int8" or sk == 1 else plan[2] == 1, kind
        _check_epilogues(nat, cuda_device, kind, Bw, Bw, M, N, K)


@pytest.mark.parametrize("N,K", [(2048, 8192), (944, 4240), (2064, 4096), (4096, 1024)])
def test_fp8_row_has_the_same_bits_in_every_call(nat, cuda_device, N, K):
    """One fp32 accumulator per element, whatever tiles the call's M and N choose: a row alone, among others or in a
    batch, and a column of separate or stacked weights, have the same bits."""
    g = Hp.gen(N + K)
    d = cuda_device
    a = torch.randn(1100, K, generator=g).to(E4M3).to(d)
    w = torch.randn(N, K, generator=g).to(E4M3).to(d)
    sa = (torch.rand(1100, generator=g) * 0.01 + 0.001).to(d)
    sw = (torch.rand(N, generator=g) * 0.01 + 0.001).to(d)
    full = nat.fp8_mm(a, w, sa, sw, False, torch.bfloat16)[0].cpu()
    for m in (1, 36, 128, 256, 512, 1024):
        Hp.assert_bit_equal(nat.fp8_mm(a[:m], w, sa[:m], sw, False, torch.bfloat16)[0], full[:m], f"{m} rows")
    for n in (16, 464, N // 32 * 16):
        for m in (128, 300):
            Hp.assert_bit_equal(nat.fp8_mm(a[:m], w[:n], sa[:m], sw[:n], False, torch.bfloat16)[0], full[:m, :n].contiguous(),
                                f"{m} rows, {n} columns")
    batch = nat.fp8_mm(a[:96].view(3, 32, K), w, sa[:96].view(3, 32), sw, False, torch.bfloat16)
    Hp.assert_bit_equal(batch.reshape(96, N), full[:96], "a batch")


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("B,Bw,M,N,K", [(1, 1, 37900, 64, 144), (1, 1, 38000, 128, 272), (40, 40, 100, 1040, 1040),
                                        (160, 160, 128, 128, 1024), (7, 1, 77, 272, 400), (300, 1, 3, 144, 64), (1, 3, 33, 96, 208)])
def test_padded_pair_tiles_and_folded_batches(nat, cuda_device, kind, B, Bw, M, N, K):
    """Pair tiles half of which is padding (three rounds of them, N or M at most 128), a batch on shared weights as rows
    of one product (tiles that straddle batch entries and their gate rows), one activation on a batch of weights.
    Bounds as in _check_epilogues."""
    qd = torch.int8 if kind == "int8" else E4M3
    d = cuda_device
    g = torch.Generator(device=d).manual_seed(M + N + K)

    def mk(*s):
        x = torch.randint(-127, 128, s, generator=g, device=d) if kind == "int8" else torch.randn(s, generator=g, device=d)
        return x.to(qd)

    a, w = mk(B, M, K), mk(*((Bw, N, K) if Bw > 1 else (N, K)))
    sa = torch.rand(B, M, generator=g, device=d) * 0.01 + 0.001
    sw = torch.rand(*((Bw, N) if Bw > 1 else (N,)), generator=g, device=d) * 0.01 + 0.001
    bias = torch.randn(N, generator=g, device=d) * 0.1
    mmb = nat.q8_mm_bias if kind == "int8" else nat.fp8_mm_bias
    out = mmb(a, w, bias, sa, sw, False, torch.bfloat16)
    assert out.shape == (max(B, Bw), M, N)
    for i in range(0, max(B, Bw), max(1, max(B, Bw) // 8)):
        ai, si = a[min(i, B - 1)], sa[min(i, B - 1)]
        wi, swi = (w[i], sw[i]) if Bw > 1 else (w, sw)
        y = (ai.double() @ wi.double().T) * si.double().unsqueeze(-1) * swi.double() + bias.double()
        assert bool(((out[i].double() - y).abs() <= 2.0 ** -8 * y.abs() + 2e-6 * y.abs().max()).all())
    if Bw == 1:
        gate = torch.randn(B, 1, N, generator=g, device=d).to(torch.bfloat16)
        resid = torch.randn(B, M, N, generator=g, device=d).to(torch.bfloat16)
        fused = nat.mm_gate_residual(a, w, bias, sa, sw, gate, resid)
        Hp.assert_bit_equal(fused, gate * out + resid, "gate and residual in the epilogue")


@pytest.mark.parametrize("M,N,K", [(6144, 2048, 2048),            # 13 tiles of 160 columns for each of 6 row blocks
                                   (6100, 2000, 2064),            # M, N and K tails, the last narrow tile partial
                                   (2002, 6144, 2048), (3096, 2048, 4112), (12510, 2048, 2048), (7401, 2048, 4096)])
@pytest.mark.parametrize("kind", ["int8", "fp8", "fp8 e4m3 out", "int8 gelu", "int8 residual", "fp8 residual"])
def test_narrow_tiles_of_the_last_round(cuda_device, M, N, K, kind):
    """Products whose last round is cut into narrow tiles: every row has the bits that it has in a call of few rows (other
    tiles on the other kernel), where int8 sums are exact and fp8 sums have one order."""
    from q8_kernels_b200 import native as nat
    g = torch.Generator(device=cuda_device).manual_seed(M + N + K)
    if kind.startswith("int8"):
        a, b = (torch.randint(-127, 128, s, generator=g, device=cuda_device, dtype=torch.int8) for s in ((M, K), (N, K)))
    else:
        a, b = (torch.randn(s, generator=g, device=cuda_device).to(torch.float8_e4m3fn) for s in ((M, K), (N, K)))
    sa, sb = torch.rand(M, generator=g, device=cuda_device) / K, torch.rand(N, generator=g, device=cuda_device)
    bias = torch.randn(N, generator=g, device=cuda_device)
    resid = torch.randn(1, M, N, generator=g, device=cuda_device).to(torch.bfloat16)
    gate = torch.randn(1, 1, N, generator=g, device=cuda_device).to(torch.bfloat16)
    out = torch.float8_e4m3fn if "e4m3" in kind else torch.bfloat16

    def product(r):
        if "residual" in kind:
            return nat.mm_gate_residual(a[r], b, bias, sa[r], sb, gate, resid[:, r])
        mm = nat.q8_mm_bias if kind.startswith("int8") else nat.fp8_mm_bias
        return mm(a[r], b, bias, sa[r], sb, "gelu" in kind, out)
    got = product(slice(0, M))[0]
    for r0 in range(0, M, 512):
        r = slice(r0, min(r0 + 512, M))
        want = product(r)[0]
        assert torch.equal(got[r].view(torch.uint8), want.view(torch.uint8)), (r0, (got[r] != want).sum())


_NARROW = [(6144, 2048, 2048, 160), (6100, 2000, 2064, 160), (2002, 6144, 2048, 160), (3096, 2048, 4112, 128), (12510, 2048, 2048, 96),
           (7401, 2048, 4096, 64)]
_EDGES = [(2560, 2048, 2048, 32), (2400, 2000, 4112, 32), (4800, 1024, 2048, 32),    # half of the epilogue warps have no column
          (7296, 1024, 2064, 192), (7500, 1008, 4112, 192)]


@pytest.mark.parametrize("M,N,K,bn,kind", [c + (k,) for c in _EDGES for k in ("int8", "fp8", "fp8 e4m3 out", "int8 gelu")]
                         + [(m, n, max(k, 4112), bn, r) for m, n, k, bn in _NARROW + _EDGES for r in ("int8 residual", "fp8 residual")])
def test_every_width_of_the_last_round(cuda_device, M, N, K, bn, kind):
    """The narrowest and the widest tiles too, and the residual tail at the K from which its last round is cut; the width that
    148 SMs give is asserted."""
    import ctypes
    from q8_kernels_b200 import _lib
    plan, columns = (ctypes.c_int * 3)(), ctypes.c_int()
    assert _lib.lib.q8k_mm_plan(int(kind.startswith("int8")), 1, 1, M, N, K, ctypes.cast(plan, ctypes.c_void_p)) == 0
    assert _lib.lib.q8k_mm_last_round_columns(1, 1, M, N, K, int("residual" in kind), ctypes.cast(ctypes.byref(columns), ctypes.c_void_p)) == 0
    assert (plan[0], columns.value) == (1, bn)
    test_narrow_tiles_of_the_last_round(cuda_device, M, N, K, kind)
    assert _lib.read_status(cuda_device) == 0
