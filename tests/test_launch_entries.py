"""The way from Python to the kernels' entry points (native/csrc/launch.cc): every signature against the sources, what an
argument becomes, what a refusal raises, and the products that are checked, allocated and launched in one go."""
import copy
import ctypes
import glob
import os
import re
import subprocess
import sys

import pytest
import torch

from rllm_b200.kernels import build, ops

LETTERS = {"int": "i", "long long": "l", "float": "f"}


def prototypes():
    """Entry point -> (library, letters of its arguments ahead of the stream), as the sources declare them."""
    found = {}
    for path in glob.glob(os.path.join(build.CSRC, "*.cu")):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for name, args in re.findall(r"RLLM_EXPORT int (rllm_\w+)\(([^)]*)\)\s*\{", text):
            letters = ""
            args = [re.sub(r"\s+", " ", a).strip() for a in args.split(",")]
            if args[-1] != "cudaStream_t stream":
                continue
            for a in args[:-1]:
                letters += "p" if "*" in a else LETTERS.get(re.sub(r"^const ", "", a.rsplit(" ", 1)[0]), "?")
            found[name] = (os.path.basename(path)[:-3], letters)
    return found


def test_signatures_are_those_of_the_sources():
    have = prototypes()
    for symbol, (library, letters, what) in ops._TABLE.items():
        assert have[symbol] == (library, letters), symbol
        assert what and getattr(ops._entries, symbol) is getattr(ops._entries, symbol)          # compiled, and made once


def test_what_is_refused_before_anything_is_called():
    x = torch.zeros(2, 2)
    with pytest.raises(ops.KernelError, match="CUDA tensors only"):
        ops._entries.rllm_residual_add(x, x, 0, 4)
    with pytest.raises(TypeError, match="tensor or None"):
        ops._entries.rllm_residual_add(None, 3, 0, 4)
    with pytest.raises(TypeError, match="4 arguments"):
        ops._entries.rllm_residual_add(None, None, 0)
    with pytest.raises(TypeError):
        ops._entries.rllm_residual_add(None, None, 1.5, 4)
    with pytest.raises(ValueError, match="no signature"):
        ops._launch().entry("pxp", lambda: 0, "odd")
    assert ops.product(x, x) is None and ops.product(x.bfloat16(), x.bfloat16()) is None


def test_a_name_that_is_no_entry_point_is_no_attribute():
    assert not hasattr(ops._entries, "rllm_no_such_kernel") and copy.copy(ops._entries) is not ops._entries


def test_what_the_tensor_library_throws_is_an_exception():
    """A tensor without memory of its own to point at; in a process of its own, which an exception that leaves the C++ ends."""
    code = "import torch\nfrom rllm_b200.kernels import ops\ntry:\n    ops._launch().error_word(0, torch.eye(2).to_sparse())\n" \
           "except RuntimeError as e:\n    print('raised')\n"
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert done.returncode == 0 and done.stdout == "raised\n", done.stderr[-500:]


@pytest.mark.gpu
def test_what_the_arguments_become_and_what_a_refusal_raises():
    seen = []
    answer = [0]
    proto = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_void_p)
    callback = proto(lambda *a: (seen.append(a), answer[0])[1])
    entry = ops._launch().entry("ppil", lambda: ctypes.cast(callback, ctypes.c_void_p).value, "odd")
    t = torch.zeros(8, device="cuda")
    before = ops.LAUNCHES[0]
    entry(t[2:], None, True, -(1 << 40))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        entry(None, t, (1 << 32) + 5, 7)                   # an int is the low 32 bits, as ctypes has it
    main = torch.cuda.current_stream().cuda_stream or None
    assert seen == [(t.data_ptr() + 8, None, 1, -(1 << 40), main), (None, t.data_ptr(), 5, 7, side.cuda_stream)]
    assert ops.LAUNCHES[0] == before + 2
    for code, text in ((-1, "odd: refused its arguments"), (-2, "odd: this size is legal but no kernel"), (719, "odd: CUDA error 719")):
        answer[0] = code
        with pytest.raises(ops.KernelError, match=text):
            entry(None, None, 0, 0)


@pytest.mark.gpu
def test_products_that_cannot_be_made_raise():
    ops.gemm_error_word(torch.device("cuda", 0))
    x = torch.randn(4, 64, device="cuda").bfloat16()
    for a, b in ((x.to_sparse_csr(), x), (x, x.to_sparse_csr())):      # (no strides)
        with pytest.raises(RuntimeError):
            ops.product(a, b)
    assert ops.product(x, torch.nn.Parameter(x)) is not None
    with pytest.raises(torch.OutOfMemoryError):            # 2^22 x 2^16 results
        ops.product(torch.zeros(1 << 22, 8, device="cuda", dtype=torch.bfloat16), torch.zeros(1 << 16, 8, device="cuda", dtype=torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,f32,silu", [(1, 40, 64, False, False), (8, 136, 2048, True, False), (5, 64, 256, False, True),
                                            (9, 40, 64, False, False), (2048, 2100, 136, False, False), (1500, 4096, 72, False, True)])
def test_products_in_one_go_are_the_products(M, N, K, f32, silu, monkeypatch):
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N * (2 if silu else 1), K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    ops.gemm_error_word(x.device)
    got = ops.product(x, w, f32, silu, (7.0, 1.5, 0.5) if silu else ops.PLAIN_GATE)
    takes = ops.small_m_takes(x, w) or ops.tcgen05_takes(x, w, silu=silu)
    assert (got is not None) == takes
    if takes:
        want = torch.empty(M, N, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
        call = ops.gemm_small_m if ops.small_m_takes(x, w) else ops.gemm_tcgen05
        call(x, w, want, "silu_mul" if silu else "store", gate=(7.0, 1.5, 0.5) if silu else ops.PLAIN_GATE)
        assert got.dtype is want.dtype and torch.equal(got, want)
    room = torch.zeros(max(M * K, w.numel()) + 8, device="cuda", dtype=torch.bfloat16)
    off = lambda t: room[1:1 + t.numel()].view_as(t).copy_(t)  # noqa: E731
    if M > ops.SMALL_M_MAX:                                # off 16 bytes: TMA does not take it
        assert not ops.tcgen05_takes(off(x), w, silu=silu) and ops.product(room[1:1 + x.numel()].view_as(x), w, f32, silu) is None
        assert not ops.tcgen05_takes(x, off(w), silu=silu) and ops.product(x, room[1:1 + w.numel()].view_as(w), f32, silu) is None
    else:                                                  # the kernel refuses it
        a = off(x)
        with pytest.raises(ops.KernelError):
            ops.product(a, w, f32, silu)
        with pytest.raises(ops.KernelError):
            ops.gemm_small_m(a, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), "silu_mul" if silu else "store")
    for odd in (x[:, :K - 8], x.float(), x.t(), x.cpu(), x[None]):
        assert ops.product(odd, w, f32, silu) is None
    monkeypatch.setenv("RLLM_GEMM", "library")
    assert ops.product(x, w, f32, silu) is None
    monkeypatch.setenv("RLLM_GEMM", "tcgen05")
    assert ops.product(x, w, f32, silu) is not None
    monkeypatch.setenv("RLLM_GEMM", "no_tcgen05")
    assert (ops.product(x, w, f32, silu) is not None) == (M <= ops.SMALL_M_MAX)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,silu", [(128 * 12, 256 * 8, False), (128 * 12 - 127, 256 * 7 + 1, False), (128 * 11, 256 * 8, False), (128 * 95, 256, False),
                                      (128 * 96, 256, False), (128 * 12, 128 * 8, True), (128 * 12, 128 * 7, True), (8, 65537, False), (8, 65536, False), (9, 65537, False)])
@pytest.mark.parametrize("head", ["", "library"])
def test_products_in_one_go_follow_the_rule(M, N, silu, head, monkeypatch):
    """Both sides of the fewest tiles and of the tallest weight that takes few rows whatever the head's switch says."""
    monkeypatch.setenv("RLLM_HEAD", head)
    x = torch.zeros(M, 16, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(N * (2 if silu else 1), 16, device="cuda", dtype=torch.bfloat16)
    ops.gemm_error_word(x.device)
    takes = (ops.small_m_takes(x, w) or ops.tcgen05_takes(x, w, silu=True)) if silu else ops.gemm_bf16(x, w, torch.bfloat16) is not None
    assert (ops.product(x, w, silu=silu) is not None) == takes
