"""The native form of the Python boundary (`_host`): what it takes, what it hands back, what it leaves to the Python code.
On the CPU, with objects that have a tensor's attributes and a stand-in for the library's `run`."""
import ctypes
import os
import sysconfig
import warnings

import pytest
import torch

from radeonflow_kernels_b200 import _lib, build, gemm, moe

FP8, F32, BF16, F16 = torch.float8_e4m3fn, torch.float32, torch.bfloat16, torch.float16


class Fake:
    def __init__(self, shape, dtype, ptr, is_cuda=True, contiguous=True):
        self.shape, self.dtype, self.is_cuda = torch.Size(shape), dtype, is_cuda
        self._ptr, self._contiguous = ptr, contiguous

    def is_contiguous(self):
        return self._contiguous

    def data_ptr(self):
        return self._ptr


@pytest.fixture
def host(rf_lib):
    """The module with a `run` that records its arguments; afterwards it is the library's again."""
    h = _lib.host()
    calls = []
    kind = ctypes.CFUNCTYPE(None, *[ctypes.c_void_p] * 5, *[ctypes.c_int] * 3, *[ctypes.c_void_p] * 2)
    run = kind(lambda *a: calls.append(a))
    h.setup(ctypes.cast(run, ctypes.c_void_p).value, lambda: 3, lambda dev: 0x700 + dev, FP8, F32, BF16, F16)
    yield h, calls
    _lib._host = None
    _lib.host()


def _operands(m=48, n=192, k=384):
    return [Fake((m, k), FP8, 0x10), Fake((n, k), FP8, 0x20), Fake((m, k // 128), F32, 0x30),
            Fake(((n + 127) // 128, k // 128), F32, 0x40), Fake((m, n), BF16, 0xFFFF000000000050)]


def test_gemm_passes_addresses_sizes_and_the_current_stream(host):
    h, calls = host
    assert h.gemm(*_operands()) is True
    assert calls == [(0x10, 0x20, 0x30, 0x40, 0xFFFF000000000050, 48, 192, 384, None, 0x703)]


@pytest.mark.parametrize("i,change", [
    (0, {"is_cuda": False}), (4, {"is_cuda": False}), (1, {"contiguous": False}), (3, {"contiguous": False}),
    (0, {"dtype": torch.uint8}), (1, {"dtype": torch.float8_e4m3fnuz}), (2, {"dtype": torch.float64}), (4, {"dtype": F16}),
    (0, {"shape": (48, 385)}), (1, {"shape": (192, 256)}), (2, {"shape": (48, 4)}), (3, {"shape": (1, 3)}),
    (4, {"shape": (192, 48)}), (0, {"shape": (48 * 384,)}), (4, {"shape": (1, 48, 192)})])
def test_gemm_leaves_every_other_form_alone(host, i, change):
    h, calls = host
    ops = _operands()
    t = dict(shape=ops[i].shape, dtype=ops[i].dtype, ptr=ops[i]._ptr)
    t.update(change)
    ops[i] = Fake(**t)
    assert h.gemm(*ops) is False and calls == []
    assert h.gemm(*ops[:4]) is False


def test_gemm_passes_exceptions_on(host):
    h, calls = host
    with pytest.raises(AttributeError):
        h.gemm(1, 2, 3, 4, 5)
    ops = _operands()
    ops[2].data_ptr = lambda: 1 / 0
    with pytest.raises(ZeroDivisionError):
        h.gemm(*ops)
    assert calls == []


def test_fp16_addresses(host):
    h, _ = host
    w = {"a": Fake((4, 4), F16, 0x1000), "b": Fake((2,), F16, 0xFFFF000000002000), "c": Fake((2,), F32, 0x3000)}
    assert h.fp16_addresses(w, ("a", "b")) == (0x1000).to_bytes(8, "little") + (0xFFFF000000002000).to_bytes(8, "little")
    assert h.fp16_addresses(w, ()) == b""
    assert h.fp16_addresses(w, ("a", "c")) is None          # another type
    assert h.fp16_addresses(w, ("a", "d")) is None          # not there
    assert h.fp16_addresses([1], ("a",)) is None


def test_the_extension_is_named_after_its_interpreter(rf_lib):
    """... so that another one does not find it, and building for that one is not skipped as done."""
    assert build.HOST_PATH == _lib.HOST_PATH and build.HOST_PATH.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert _lib.host().__file__ == _lib.HOST_PATH and os.path.exists(build.build_host())
    assert not [f for f in os.listdir(build.PKG_DIR) if f.endswith(".tmp")]


@pytest.fixture
def no_extension(rf_lib, monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(_lib, "HOST_PATH", str(tmp_path / os.path.basename(_lib.HOST_PATH)))


def test_without_the_extension_the_python_code_serves_every_call(no_extension):
    with pytest.warns(RuntimeWarning, match="cannot be used"):
        assert _lib.host().gemm(*_operands()) is False
    with warnings.catch_warnings():
        warnings.simplefilter("error")                      # said once
        cpu = [torch.zeros(s, dtype=t) for s, t in (((16, 128), FP8), ((64, 128), FP8), ((16, 1), F32), ((1, 1), F32),
                                                    ((16, 64), BF16))]
        for call in (gemm.custom_kernel, lambda data: gemm.fp8_mm(*data)):
            with pytest.raises(ValueError, match="must be CUDA tensors"):
                call(cpu)
        w = {f"experts.{i}.1.weight": Fake((4, 4), F16, 0x1000 * (i + 1)) for i in range(3)}
        assert list(moe._expert_ptrs(w, 3, 1, ctypes.c_ulonglong)) == [0x1000, 0x2000, 0x3000]


def test_a_torch_without_cuda_gets_the_python_errors(rf_lib, monkeypatch):
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    with pytest.warns(RuntimeWarning), pytest.raises(ValueError, match="must be CUDA tensors"):
        gemm.custom_kernel([torch.zeros(1, 1)] * 5)


def test_the_library_is_built_where_the_extension_cannot_be(rf_lib, monkeypatch, capsys):
    monkeypatch.setenv("CXX", "false")
    assert build.build_host() == build.HOST_PATH            # there already
    monkeypatch.setattr(build, "HOST_PATH", build.HOST_PATH + ".other")
    assert build.build() == build.LIB_PATH and os.path.exists(build.LIB_PATH)
    assert "without its extension" in capsys.readouterr().err and not os.path.exists(build.HOST_PATH)
    monkeypatch.setenv("CXX", "no-such-compiler")
    assert build.build() == build.LIB_PATH


@pytest.mark.gpu
def test_results_without_the_extension_are_the_same_bits(rf_lib, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = (torch.randn(s, generator=g, device="cuda").to(FP8) for s in ((96, 256), (192, 256)))
    a_s, b_s = torch.rand((96, 2), generator=g, device="cuda"), torch.rand((2, 2), generator=g, device="cuda")
    c = [torch.empty((96, 192), dtype=BF16, device="cuda") for _ in range(2)]
    assert _lib.host() is not _lib._NoHost
    gemm.custom_kernel((a, b, a_s, b_s, c[0]))
    monkeypatch.setattr(_lib, "_host", _lib._NoHost)
    gemm.custom_kernel((a, b, a_s, b_s, c[1]))
    assert torch.equal(c[0].view(torch.int16), c[1].view(torch.int16)) and c[0].abs().sum() > 0
