"""CPU checks of the drop-in boundary: the native library loads, exports every
symbol the header declares, rejects bad arguments before touching the GPU, and
the Python layer mirrors the reference's API surface."""
import inspect
import os
import re

import pytest
import torch

import helpers as Hp

HEADER = os.path.join(Hp.REPO_ROOT, "include", "q8_kernels_b200.h")


def _declared_symbols():
    text = open(HEADER).read()
    return sorted(set(re.findall(r"\b(q8k_\w+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from q8_kernels_b200 import _lib
    names = _declared_symbols()
    assert len(names) >= 16
    for n in names:
        assert hasattr(_lib.lib, n), f"{n} declared in the header but not exported"
        assert n in _lib.SIGNATURES, f"{n} has no ctypes signature"
    assert _lib.lib.q8k_version() >= 100
    assert _lib.lib.q8k_error_string(-3).decode() == "workspace too small"


def test_argument_validation_without_gpu():
    """Validation happens on the host before any launch, so it is testable here."""
    from q8_kernels_b200 import _lib
    lib = _lib.lib
    buf = (torch.zeros(4096, dtype=torch.uint8).data_ptr() + 15) // 16 * 16
    # dim not a multiple of 16
    assert lib.q8k_tokenwise_quant(buf, _lib.DT_BF16, buf, _lib.DT_I8, buf, 4, 24, 24, None) == -1
    assert b"multiple of 16" in lib.q8k_last_error_detail()
    # unsupported output dtype
    assert lib.q8k_tokenwise_quant(buf, _lib.DT_BF16, buf, _lib.DT_BF16, buf, 4, 64, 64, None) == -2
    # null pointer
    assert lib.q8k_rms_norm(None, _lib.DT_BF16, None, buf, _lib.DT_BF16, None, 4, 64, None) == -1
    # Hadamard dim limit
    assert lib.q8k_fast_hadamard_transform(buf, _lib.DT_BF16, buf, _lib.DT_BF16, 1, 32768, 32768, 1.0, None) == -2
    # GEMM batch mismatch and bad N
    assert lib.q8k_q8_mm(buf, buf, None, buf, buf, buf, _lib.DT_BF16, 2, 3, 8, 16, 64, 0, None, None) == -1
    assert lib.q8k_fp8_mm(buf, buf, None, buf, buf, buf, _lib.DT_BF16, 1, 1, 8, 24, 64, 0, None, None) == -1
    # linear: workspace too small / misaligned
    need = lib.q8k_linear_workspace_bytes(128, 256)
    assert need >= 128 * 256 + 128 * 4
    ws = (buf + 255) // 256 * 256
    assert lib.q8k_linear(buf, _lib.DT_BF16, buf, _lib.DT_I8, buf, None, buf, _lib.DT_BF16, 128, 64, 256, 1, 0,
                          ws, 16, None, None) == -3
    assert lib.q8k_linear(buf, _lib.DT_BF16, buf, _lib.DT_I8, buf, None, buf, _lib.DT_BF16, 128, 64, 256, 1, 0,
                          ws + 16, need, None, None) == -1
    # zero rows is a no-op, not an error
    assert lib.q8k_tokenwise_quant(None, _lib.DT_BF16, None, _lib.DT_I8, None, 0, 64, 64, None) == 0


def test_ops_fail_loudly_on_cpu_tensors():
    import q8_kernels_b200 as q8
    x = torch.randn(4, 64).bfloat16()
    with pytest.raises(q8._lib.Q8KernelError, match="no CPU path"):
        q8.functional.quantizer.quantize(x)
    with pytest.raises(q8._lib.Q8KernelError):
        q8.functional.fast_hadamard.hadamard_transform(x)


def test_python_api_surface_matches_reference():
    import q8_kernels_b200 as q8
    F, M = q8.functional, q8.modules
    sig = lambda f: list(inspect.signature(f).parameters)  # noqa: E731
    assert sig(F.linear.q8_linear) == ["a", "b", "bias", "scale_a", "scale_b", "fuse_gelu", "out_dtype"]
    assert sig(F.linear.fp8_linear) == ["a", "b", "bias", "scale_a", "scale_b", "use_hadamard", "out_dtype"]
    assert sig(F.fast_hadamard.hadamard_transform) == ["x", "scale", "out_type"]
    assert sig(F.flash_attention.flash_attn_func)[:6] == ["q", "k", "v", "softmax_scale", "batch_mask",
                                                          "apply_qk_hadamard"]
    assert sig(F.rms_norm.rms_norm_8bit) == ["x", "weights", "out_type"]
    assert sig(F.rope.apply_rope) == ["x", "cos_freqs", "sin_freqs", "out_type"]
    assert sig(F.fma.multiply_add) == ["x", "y", "z", "scale_add"]
    assert sig(F.quantizer.quantize) == ["x"] and sig(F.quantizer.quantize_fp8) == ["x"]
    lin = M.Q8Linear(64, 32, bias=True)
    assert set(lin.state_dict()) == {"weight", "bias", "scales"}
    assert lin.weight.dtype == torch.int8 and lin.scales.dtype == torch.float32 and lin.bias.dtype == torch.float32
    f8 = M.FP8Linear(64, 32, bias=False)
    assert set(f8.state_dict()) == {"weight", "scales"} and f8.weight.dtype == torch.float8_e4m3fn
    blk = q8.blocks.LTXTransformerBlock(64, 2, 32, 64)
    keys = set(blk.state_dict())
    for k in ("scale_shift_table", "attn1.to_q.weight", "attn1.to_q.scales", "attn1.q_norm.weight",
              "attn2.to_k.bias", "attn1.to_out.weight", "ff.act.proj.weight", "ff.proj_down.scales"):
        assert k in keys, k
    assert "norm1.weight" not in keys                                      # norm_affine=False


def test_rope_table_on_cpu_matches_reference_vectors():
    """The product's RoPE table is pure torch: on the CPU it must reproduce, bit for bit, the table
    the reference's own precompute_freqs_cis produced for the golden fixture."""
    import golden_io as G
    import q8_kernels_b200 as q8
    d = G.load("ref_freqs_cis.npz")
    cos, sin = q8.blocks.precompute_freqs_cis(G.t(d["grid"]), 2048)
    Hp.assert_bit_equal(cos, G.t(d["cos"]), "cos")
    Hp.assert_bit_equal(sin, G.t(d["sin"]), "sin")
    assert torch.equal(q8.blocks.latent_grid(2, 3, 4), G.t(d["grid"]))


def _forms():
    """Contiguous, sliced, transposed, expanded, offset and empty tensors of one to four dims."""
    base = torch.arange(4 * 6 * 8 * 16, dtype=torch.float32).reshape(4, 6, 8, 16)
    yield from (base, base[0], base[0, 0], base[0, 0, 0], base[:, 1:5], base[:, :, :, :8], base[..., 8:], base.transpose(1, 2),
                base.transpose(0, 3), base[::2], base[:, ::3], base[:1].expand(5, 6, 8, 16), base[0, 0, :1].expand(7, 16),
                base.flatten()[4:4 + 160].view(10, 16), base[:0], base[:, :0], base[:, :, :1, ::2], base.permute(2, 0, 1, 3))
    yield base.to(torch.bfloat16)[:, :, :, :8]


@pytest.mark.parametrize("i", range(19))
def test_row_arguments_describe_the_same_rows_for_every_layout(i):
    """What a kernel is told (pointer, rows, dim, row stride) reads back as x.reshape(-1, dim), whether or not the
    tensor takes the contiguous shortcut."""
    from q8_kernels_b200 import native
    x = list(_forms())[i]
    want = x.reshape(-1, x.shape[-1])
    t, rows, dim, stride = native._rows(x)
    assert (rows, dim) == tuple(want.shape) and (rows <= 1 or stride >= dim)
    got = torch.as_strided(t, (rows, dim), (stride, 1), t.storage_offset())
    assert torch.equal(got, want)
    t, rows, dim = native._dense_rows(x)
    assert (rows, dim) == tuple(want.shape) and t.is_contiguous() and torch.equal(t.reshape(rows, dim), want)
    c, s, n = native._tables(x, x.clone(), dim)
    assert n == rows and c.is_contiguous() and s.is_contiguous() and torch.equal(c.reshape(rows, dim), want)


def test_gemm_plan_keeps_to_what_the_split_kernel_can_run():
    """Over sizes from one row up: tile widths are multiples of 16 (of 32 for four shares of K) up to 256, every CTA of a
    K split has at least two slabs, FP8 never splits K, and batches on shared weights are planned as rows."""
    import ctypes
    from q8_kernels_b200 import _lib
    plan, folded = (ctypes.c_int * 3)(), (ctypes.c_int * 3)()

    def ask(p, *a):
        assert _lib.lib.q8k_mm_plan(*a, ctypes.cast(p, ctypes.c_void_p)) == 0
        return tuple(p)

    for int8 in (0, 1):
        for batch in (1, 3, 64):
            for m in (1, 16, 77, 128, 129, 512, 2002, 24576):
                for n in (16, 48, 128, 144, 2048, 10240):
                    for k in (16, 256, 272, 1024, 4240, 8192):
                        pair, bn, sk = ask(plan, int8, batch, batch, m, n, k)
                        assert (pair, bn, sk) == (1, 256, 1) or (pair == 0 and bn % (32 if sk == 4 else 16) == 0 and 32 <= bn <= 256)
                        assert sk == 1 or (int8 and sk in (2, 4) and (k + 127) // 128 >= 2 * sk)
                        assert ask(plan, int8, batch, 1, m, n, k) == ask(folded, int8, 1, 1, batch * m, n, k)
    assert _lib.lib.q8k_mm_plan(1, 1, 1, 0, 16, 16, ctypes.cast(plan, ctypes.c_void_p)) != 0


def test_last_round_columns_are_what_the_pair_kernel_can_run():
    """Widths over sizes around the edges of row blocks and rounds: multiples of 32 up to 192 or the whole 256, never with a
    batch of weights or a short K, and a width that leaves one half of the epilogue warps without a column (32) is among them."""
    import ctypes
    from q8_kernels_b200 import _lib
    c = ctypes.c_int()

    def ask(*a):
        assert _lib.lib.q8k_mm_last_round_columns(*a, ctypes.cast(ctypes.byref(c), ctypes.c_void_p)) == 0
        return c.value

    widths = set()
    for m in list(range(129, 12600, 257)) + [2433, 2560, 24576]:
        for n in (128, 1008, 1024, 2048, 6144, 10240):
            for k in (2048, 2064, 4096):
                bn = ask(1, 1, m, n, k, 0)
                widths.add(bn)
                assert bn == 256 or (bn % 32 == 0 and 32 <= bn <= 192)
                assert ask(1, 1, m, n, k, 1) == (bn if k >= 4096 else 256)
                assert ask(2, 1, m, n, k, 0) == ask(1, 1, 2 * m, n, k, 0)
                assert ask(2, 2, m, n, k, 0) == ask(1, 1, m, n, 2032, 0) == 256
    assert widths == {32, 64, 96, 128, 160, 192, 256}
    assert _lib.lib.q8k_mm_last_round_columns(1, 1, 0, 16, 16, 0, ctypes.cast(ctypes.byref(c), ctypes.c_void_p)) != 0


def test_host_path_looks_at_no_argument_of_a_call_with_a_wrong_number_of_them():
    """Every function of the native host path answers None to any other number of arguments than its own (reading on behind
    the last one ended the process)."""
    from q8_kernels_b200 import _host
    arguments = {"tokenwise_quant": 2, "hadamard_quant": 3, "fast_hadamard_transform": 3, "norm_modulate_quant": 4,
                 "transpose_quant": 2, "dequant_hadamard": 3, "rms_norm": 3, "rms_norm_backward": 5, "rope": 4, "rope_backward": 4,
                 "mm": 9, "mm_gate_residual": 7, "linear": 7, "flash_attention": 7, "attention_prep_rows": 5, "qk_norm_rope_prep": 6,
                 "kv_prep": 6, "qk_norm_rope_prep_pair": 9}
    assert set(arguments) == {n for n in dir(_host) if not n.startswith(("_", "set_"))}
    x = torch.zeros(2, 16)
    for name, want in arguments.items():
        for n in list(range(want)) + [want + 1, 20]:
            for a in (x, None, True, 1.0, torch.int8):
                assert getattr(_host, name)(*[a] * n) is None, (name, n)


def test_rotary_tables_of_a_wrong_number_are_refused():
    """A sequence of tables that is not (cos, sin) reaches the Python body, which refuses it."""
    from q8_kernels_b200 import native
    x, w, c = torch.zeros(1, 4, 512, dtype=torch.bfloat16), torch.ones(512), torch.zeros(1, 4, 512)
    for freqs in ((), (c,), (c, c, c)):
        for call in (lambda: native.qk_norm_rope_prep(x, w, freqs, 8, True, 0.5),
                     lambda: native.qk_norm_rope_prep_pair(x, x, w, w, freqs, 8, True, 0.5)):
            with pytest.raises((ValueError, native.Q8KernelError)):
                call()
