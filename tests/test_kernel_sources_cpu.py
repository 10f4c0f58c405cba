"""Properties of the kernel sources that no run can show, because the case that breaks them would hang a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "cosmos_rl_b200" / "csrc"


def test_decode_softmax_warps_leave_their_loops_together():
    """The four softmax warps of the decode attention meet at a named barrier, which has no time limit. Their waits do have
    one, and may run out in some of the warps only. So a warp may leave a loop only on a value that the barrier returned to
    all four: every ``break`` follows an assignment from ``softmax_bar``, and no loop condition reads the abort flag."""
    src = (CSRC / "paged_decode_tc.cu").read_text()
    role = src[src.index("softmax / epilogue (warps 2..5)"):]
    role = role[:role.index("__syncthreads()")]
    lines = [re.sub(r"//.*", "", line).strip() for line in role.splitlines()[1:]]
    lines = [line for line in lines if line and not line.startswith("#")]
    leaving = [i for i, line in enumerate(lines) if re.search(r"\b(break|goto)\b", line)]
    assert leaving
    for i in leaving:
        assert lines[i] == "if (!ok) break;" and lines[i - 1].startswith("ok = softmax_bar("), lines[i - 1:i + 1]
    for line in lines:
        if line.startswith(("for (", "while (")):
            assert "abort_flag" not in line, line


def test_local_arrays_read_as_vectors_are_aligned():
    """An array of 2-byte values that is read as one 16-byte vector says so in its declaration: as long as it lives in
    registers nothing depends on it, but in local memory the load would be misaligned."""
    for path in sorted(CSRC.glob("*.cu*")):
        src = path.read_text()
        for name in set(re.findall(r"\*reinterpret_cast<(?:const )?uint4\*>\((\w+)\)", src)):
            for decl in re.findall(r"^.*\b__nv_bfloat16 %s\[\d+\];" % re.escape(name), src, flags=re.M):
                assert "alignas(16)" in decl, (path.name, decl.strip())


def test_rms_norm_refuses_a_residual_of_other_rows(monkeypatch):
    """The kernel reads as many residual rows as there are activations: a residual whose values do not make rows of that
    length never reaches it, with gradients or without. (Tensors that only say that they are on a GPU.)"""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cosmos_rl_b200.ops import functional as F
    seen = []

    def launch(x2, weight, eps, res2, rstd):
        seen.append(tuple(res2.shape))
        return torch.empty_like(x2), torch.empty_like(x2)
    monkeypatch.setattr(F, "_rmsnorm_fwd", launch)
    with FakeTensorMode():
        make = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")
        x, weight = make(4, 512), make(512)
        for w in (weight, weight.clone().requires_grad_(True)):
            for shape in ((4, 512), (2, 2, 512), (2, 1024), (2048,)):
                F.rms_norm(x, w, residual=make(*shape))
            for shape in ((3, 500), (4, 511), (3, 2, 500)):
                with pytest.raises(RuntimeError):
                    F.rms_norm(x, w, residual=make(*shape))
    assert seen == [(4, 512)] * 8


def test_launchers_refuse_what_cannot_be_launched():
    """Wrong counts and types, sizes beyond the argument's, and tensors that have no memory end in an exception before a launch."""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cosmos_rl_b200.ops import build, native
    if not (native.available() and build.host_path().exists()):
        pytest.skip("the kernel library is not built")
    H, x = native.host(), torch.zeros(4, 8, dtype=torch.bfloat16)
    for args in ((x,), (x, 0, 0), (1, 0), (None, 0)):
        with pytest.raises(TypeError):
            H.swiglu_fwd(*args)
    with pytest.raises(TypeError):
        H.b200_swiglu_fwd(x, "out", 4, 4, None, 0)
    with pytest.raises(ValueError):
        H.b200_swiglu_fwd(x, x, 4, 1 << 31, None, 0)
    with pytest.raises(AssertionError):
        H.swiglu_fwd(x[0], 0)
    with pytest.raises(AssertionError):
        H.gemm(x, x, False, False, None, False, False, None, False, 0, None, -1, 0, 148, 0)      # not on a GPU
    with FakeTensorMode(), pytest.raises(RuntimeError, match="without memory"):
        H.swiglu_fwd(torch.empty(4, 8, dtype=torch.bfloat16, device="cuda"), 0)


def test_gated_mlp_of_mismatched_shapes_goes_through_the_checked_calls(monkeypatch):
    """The fused form hands the launcher one contraction for the activations and the weight: shapes that do not fit never reach it,
    with few rows or many. (Tensors that only say that they are on a GPU.)"""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cosmos_rl_b200.ops import build, native
    from cosmos_rl_b200.ops import functional as F
    if not (native.available() and build.host_path().exists()):
        pytest.skip("the kernel library is not built")
    fused, separate = [], []
    monkeypatch.setattr(F._GatedMLPIn, "apply", lambda x, w: (fused.append(tuple(x.shape)), None))
    monkeypatch.setattr(F._GatedMLPOut, "apply", lambda *a: None)
    monkeypatch.setattr(F, "linear_tc", lambda x, w, *b: separate.append(tuple(x.shape)))
    monkeypatch.setattr(F, "swiglu", lambda gu: torch.empty(1))
    with FakeTensorMode():
        make = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda", requires_grad=True)
        for rows in (8, 512, 1000):
            for width, gate_up, down in ((72, (96, 64), (64, 48)), (56, (96, 64), (64, 48)), (64, (96, 64), (64, 56))):
                F.gated_mlp(make(rows, width), make(*gate_up), make(*down))
                assert not fused and separate.pop(0) == (rows, width) and len(separate) == 1
                separate.clear()
        F.gated_mlp(make(512, 64), make(96, 64), make(64, 48))
    assert fused == [(512, 64)] and not separate


def test_shared_memory_of_the_norms_is_raised_on_every_device():
    """The limit of a kernel's dynamic shared memory belongs to a device: what remembers that it has been raised is kept per device,
    or the first launch on a second one fails."""
    src = (CSRC / "elementwise.cu").read_text()
    calls = [m.start() for m in re.finditer(r"cudaFuncSetAttribute\(", src)]
    assert calls and not re.search(r"static bool \w+ =", src)
    for at in calls:
        assert re.search(r"if \(!(\w+)\[dev\]\)", src[:at]) and "cudaGetDevice(&dev)" in src[:at]


def test_kernels_that_work_in_place_promise_no_separate_memory():
    """Where a launcher may pass one buffer as source and as destination, a kernel's parameters for the two are not __restrict__:
    the compiler could read what has been overwritten."""
    src = (CSRC / "elementwise.cu").read_text()
    assert "launch_rope_vec(q, k, q, k," in src
    params = re.search(r"^rope_vec_kernel\((.*?)\) \{", src, flags=re.M | re.S).group(1)
    for name in ("q", "k", "q_out", "k_out"):
        assert re.search(r"__nv_bfloat16\* %s\b" % name, params), name


def test_short_contractions_stay_whole_where_their_rows_are_on_the_128_byte_grid():
    """Whether a projection of few rows is cut is known before anything is launched: a call that is, and has no workspace, says so."""
    import pytest

    from cosmos_rl_b200.ops import native
    if not native.available():
        pytest.skip("the kernel library is not built")
    L = native.lib()

    def asks(M, N, K, ldx, ldw):
        return L.b200_skinny_linear(None, None, None, 0, None, None, 0, M, N, K, ldx, ldw, N, None, 148, None) == native.NEED_WORKSPACE

    for M in (1, 57, 256):
        for N in (72, 1024):
            assert L.b200_gemm_skinny_splits(M, N, 712, 0, 148) > 1
            for K in (704, 1000, 1032, 1088):
                assert asks(M, N, K, K, K) == (K > 704)
            for K, ldx, ldw in ((768, 776, 768), (1024, 1024, 1032), (712, 768, 768)):
                assert asks(M, N, K, ldx, ldw)
            for K in (704, 768, 1024):
                assert not asks(M, N, K, K, K) and not asks(M, N, K, K + 64, K)
            assert not asks(M, N, 696, 776, 696)


def test_the_output_heads_chunk_is_what_was_asked_for():
    """B200RL_DLOGITS_CHUNK bounds the memory of the head's backward: for any number of rows it is the number of columns held."""
    import os
    import subprocess
    import sys
    show = "from cosmos_rl_b200.ops import functional as F; print([F._dlogits_chunk(T, 152064) for T in (1, 700, 2048, 8192)])"
    env = {k: v for k, v in os.environ.items() if k != "B200RL_DLOGITS_CHUNK"}
    for extra, want in (({}, [65536, 32768, 16384, 16384]), ({"B200RL_DLOGITS_CHUNK": "4096"}, [4096] * 4),
                        ({"B200RL_DLOGITS_CHUNK": "16384"}, [16384] * 4), ({"B200RL_DLOGITS_CHUNK": "200000"}, [152064] * 4)):
        out = subprocess.run([sys.executable, "-c", show], env={**env, **extra}, cwd=CSRC.parent.parent, capture_output=True, text=True)
        assert out.returncode == 0 and out.stdout.strip() == str(want), (extra, out.stdout, out.stderr)


def test_output_head_forms():
    """CTA pairs of the output head have tiles of 256 rows: not for rows that fill half of their last one, unless the contraction is
    long enough to make up for it, and never for 128 rows or fewer."""
    from cosmos_rl_b200.ops import functional as F
    for T, V, H, pairs in ((1, 152064, 3584, False), (128, 152064, 3584, False), (129, 152064, 3584, True), (384, 152064, 3584, False),
                           (384, 32000, 512, False), (640, 32000, 512, False), (1024, 128256, 512, True), (800, 152064, 4096, True),
                           (2048, 152064, 3584, True), (300, 1500, 512, False), (5000, 152064, 3584, True)):
        ns, got = F._logprob_form(T, V, H, 148)
        assert got is pairs and 1 <= ns <= -(-V // 256), (T, V, H)


def _in_a_child(code):
    """What ``code`` prints in a process of its own, which a fault on the host would end."""
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", code], cwd=CSRC.parent.parent, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    return r.stdout.strip()


def test_rotary_embedding_of_no_heads_is_refused():
    """Without heads, or of no columns, there is nothing to divide among threads: the launcher says so."""
    import pytest

    from cosmos_rl_b200.ops import native
    if not native.available():
        pytest.skip("the kernel library is not built")
    for hq, d in ((0, 16), (0, 128), (2, 0)):
        assert int(_in_a_child("from cosmos_rl_b200.ops import native\n"
                               f"print(native.lib().b200_rope_inplace(4096, None, 4096, 4, {hq}, 0, {d}, 64, 0, 1e4, 0, None))")) < 0


def test_attention_without_kv_heads_raises():
    """Keys of no heads, on tensors that only say that they are on a GPU: an exception, as Python's own division has it."""
    import pytest

    from cosmos_rl_b200.ops import build, native
    if not (native.available() and build.host_path().exists()):
        pytest.skip("the kernel library is not built")
    assert _in_a_child("""
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from cosmos_rl_b200.ops import attention
with FakeTensorMode():
    make = lambda heads: torch.empty(4, heads, 128, dtype=torch.bfloat16, device="cuda")
    print(attention.native_flash_supported(make(8), make(4), make(4)), attention.native_flash_supported(make(8), make(3), make(3)))
    try:
        attention.native_flash_supported(make(8), make(0), make(0))
    except ZeroDivisionError:
        print("raised")
""").split() == ["True", "False", "raised"]


def test_flash_fwd_takes_its_longest_sequence_as_a_number_of_any_kind(monkeypatch):
    import types

    import numpy as np
    import torch

    from cosmos_rl_b200.ops import attention, native
    seen = []
    monkeypatch.setattr(native, "host", lambda: types.SimpleNamespace(flash_fwd=lambda *a: seen.append(a[5]) or (None, None)))
    for name in ("status_word", "num_sms"):
        monkeypatch.setattr(native, name, lambda d: 0)
    monkeypatch.setattr(native, "stream", lambda: 0)
    t = torch.zeros(1)
    for longest in (7, 7.0, np.float32(7.0), np.int64(7), torch.tensor(7), torch.tensor(7.0)):
        attention.flash_fwd(t, t, t, t, t, longest, 1.0)
    assert seen == [7] * 6 and all(type(n) is int for n in seen)


def test_native_code_is_available_when_both_libraries_are(monkeypatch, tmp_path):
    """The kernels' library alone runs nothing: its entry points are in the extension beside it."""
    from cosmos_rl_b200.ops import build, native
    assert native._LIB_PATH.parent / build.HOST_NAME == build.host_path()
    monkeypatch.setattr(native, "_LIB_PATH", tmp_path / build.LIB_NAME)
    assert not native.available()
    (tmp_path / build.LIB_NAME).touch()
    assert not native.available()
    (tmp_path / build.HOST_NAME).touch()
    assert native.available()


def test_rms_norm_refuses_a_residual_of_fewer_rows(monkeypatch):
    """Rows of the right length that are too few would be read past their end, with gradients or without. (Tensors that only say
    that they are on a GPU.)"""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cosmos_rl_b200.ops import functional as F
    monkeypatch.setattr(F, "_rmsnorm_fwd", lambda x2, weight, eps, res2, rstd: (torch.empty_like(x2), torch.empty_like(x2)))
    with FakeTensorMode():
        make = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")
        for w in (make(512), make(512).requires_grad_(True)):
            for shape in ((1, 512), (3, 512), (0, 512), (512,), (1, 3, 512)):
                with pytest.raises(RuntimeError):
                    F.rms_norm(make(4, 512), w, residual=make(*shape))
                with pytest.raises(RuntimeError):
                    F.rms_norm(make(2, 2, 512), w, residual=make(*shape))
            F.rms_norm(make(2, 2, 512), w, residual=make(4, 512))


def test_projections_of_few_rows_refuse_a_contraction_of_two_lengths(monkeypatch):
    """The launchers are told one contraction: activations that are wider than the weight would be read past its rows. (Tensors that
    only say that they are on a GPU.)"""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cosmos_rl_b200.ops import build, native
    from cosmos_rl_b200.ops import functional as F
    if not (native.available() and build.host_path().exists()):
        pytest.skip("the kernel library is not built")
    for name, value in (("status_word", None), ("num_sms", 148)):
        monkeypatch.setattr(native, name, lambda d, value=value: value)
    monkeypatch.setattr(native, "stream", lambda: 0)
    with FakeTensorMode():
        make = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")
        pos, slots = (torch.empty(4, dtype=t, device="cuda") for t in (torch.int64, torch.int32))
        for width in (56, 72):
            for call in (lambda x: F.gemm_skinny(x, make(96, 64)), lambda x: F.linear_infer(x, make(96, 64)),
                         lambda x: F.skinny_gate_up_swiglu(x, make(96, 64)),
                         lambda x: F.skinny_linear_residual_rmsnorm(x, make(96, 64), None, make(96), 1e-6),
                         lambda x: F.skinny_qkv_rope_append(x, make(96, 64), None, pos, slots, 1e4, 4, 1, 16, make(1, 2, 1, 128, 16), True)):
                with pytest.raises(AssertionError):
                    call(make(4, width))


def test_weights_elsewhere_are_not_given_to_a_kernel():
    """A weight that was left on the host, or is on another GPU, goes to torch's own product, which says so."""
    import pytest
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from cosmos_rl_b200.ops import build, native
    from cosmos_rl_b200.ops import functional as F
    if not (native.available() and build.host_path().exists()):
        pytest.skip("the kernel library is not built")
    with FakeTensorMode():
        make = lambda device, *shape: torch.empty(*shape, dtype=torch.bfloat16, device=device)
        assert F._tc_ok(make("cuda:0", 4, 64), make("cuda:0", 96, 64))
        for device in ("cpu", "cuda:1"):
            assert not F._tc_ok(make("cuda:0", 4, 64), make(device, 96, 64))
            with pytest.raises(RuntimeError, match="device"):
                F.linear_tc(make("cuda:0", 4, 64), make(device, 96, 64))
