"""CPU tests of the C-ABI boundary: the library loads, exports every symbol the header declares,
and rejects bad arguments before touching the GPU."""
import ctypes
import os
import re
import subprocess
import sys

import pytest
import torch

from radeonflow_kernels_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_functions():
    names = []
    for fn in sorted(os.listdir(os.path.join(ROOT, "include"))):
        if not fn.endswith(".h"):
            continue
        src = open(os.path.join(ROOT, "include", fn)).read()
        src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
        for m in re.finditer(r"^[A-Za-z_][\w \*]*?[\s\*]([A-Za-z_]\w*)\s*\(", src, flags=re.M):
            name = m.group(1)
            if name not in ("defined",):
                names.append(name)
    return names


def test_header_declares_the_reference_entry_points():
    names = declared_functions()
    assert "run" in names and "rf_fp8_gemm" in names


def test_every_declared_symbol_is_exported(rf_lib):
    missing = [n for n in declared_functions() if not hasattr(rf_lib, n)]
    assert not missing, missing


def test_version_string(rf_lib):
    assert b"sm_100a" in rf_lib.rf_version()


def test_perfmetrics_layout_matches_reference():
    # tests/checker/metrics.h:4-13: char[20] + 2 floats = 28 bytes; int count + 20 entries
    assert ctypes.sizeof(_lib.PerfMetricEntry) == 28
    assert ctypes.sizeof(_lib.PerfMetrics) == 4 + 20 * 28


def test_bad_arguments_are_rejected_on_the_host(rf_lib):
    buf = (ctypes.c_char * 4096)()
    p = ctypes.addressof(buf)
    p16 = (p + 15) & ~15
    args = lambda m, n, k: (p16, p16, p16, p16, p16, m, n, k, 0, None, 0, None)
    assert rf_lib.rf_fp8_gemm(*args(128, 100, 128)) == 1      # n % 64 != 0
    assert rf_lib.rf_fp8_gemm(*args(128, 128, 100)) == 1      # k % 128 != 0
    assert rf_lib.rf_fp8_gemm(*args(0, 128, 128)) == 1
    assert rf_lib.rf_fp8_gemm(None, p16, p16, p16, p16, 128, 128, 128, 0, None, 0, None) == 2
    assert rf_lib.rf_fp8_gemm(p16 + 1, p16, p16, p16, p16, 128, 128, 128, 0, None, 0, None) == 3
    assert rf_lib.rf_fp8_gemm_workspace_bytes(128, 128, 1024, 4) == 4 * 128 * 128 * 4
    assert rf_lib.rf_fp8_gemm_workspace_bytes(128, 128, 1024, 1) == 0
    assert rf_lib.rf_fp8_gemm_workspace_bytes(128, 100, 1024, 4) == 0
    # at most 64 K slices, and at most one per K block
    assert rf_lib.rf_fp8_gemm_workspace_bytes(128, 128, 128 * 100, 100) == 64 * 128 * 128 * 4
    assert rf_lib.rf_fp8_gemm_workspace_bytes(128, 128, 1024, 100) == 8 * 128 * 128 * 4
    assert rf_lib.rf_fp8_gemm_workspace_bytes(128, 128, 1024, -2) == 0      # below RF_SPLIT_STREAMK: invalid


def test_public_header_compiles_as_c_and_cpp(tmp_path):
    """include/rf_b200.h is what a C or C++ caller of the reference binds against: plain C99, no CUDA headers."""
    import shutil
    import subprocess
    hdr = os.path.join(ROOT, "include", "rf_b200.h")
    for compiler, std, ext in (("gcc", "-std=c99", "c"), ("g++", "-std=c++17", "cpp")):
        if not shutil.which(compiler):
            continue
        src = tmp_path / f"t.{ext}"
        src.write_text(f'#include "{hdr}"\nint main(void) {{ PerfMetrics m; m.count = 0; return RF_OK + m.count; }}\n')
        res = subprocess.run([compiler, std, "-Wall", "-Wextra", "-pedantic", "-Werror", "-c", str(src), "-o",
                              str(tmp_path / f"t_{ext}.o")], capture_output=True, text=True)
        assert res.returncode == 0, res.stderr


def test_expert_parallel_entries_validate_on_the_host(rf_lib):
    """The multi-GPU entry points reject bad arguments before any device work (no GPU needed)."""
    buf = (ctypes.c_char * 4096)()
    p16 = (ctypes.addressof(buf) + 15) & ~15
    ptrs = (ctypes.c_void_p * 8)(*([p16] * 8))
    # scatter GEMM: null tables, bad world, n_dim % 64
    assert rf_lib.rf_moe_grouped_gemm_scatter(p16, 128, ptrs, p16, 1, 128, 128, None, ptrs, 2, None) == 2
    assert rf_lib.rf_moe_grouped_gemm_scatter(p16, 128, ptrs, p16, 1, 128, 128, p16, None, 2, None) == 2
    assert rf_lib.rf_moe_grouped_gemm_scatter(p16, 128, ptrs, p16, 1, 128, 128, p16, ptrs, 9, None) == 1
    assert rf_lib.rf_moe_grouped_gemm_scatter(p16, 128, ptrs, p16, 1, 100, 128, p16, ptrs, 2, None) == 1
    # dispatch: experts not divisible by the ranks, rank out of range, missing pointer
    d = lambda **kw: rf_lib.rf_moe_ep_dispatch(
        kw.get("x", p16), p16, p16, p16, p16, 64, 256, 128, kw.get("e", 8), kw.get("rank", 0), kw.get("world", 2),
        kw.get("cap", 512), ptrs, kw.get("meta", ptrs), p16, p16, None, None)
    assert d(e=7) == 1 and d(rank=2) == 1 and d(world=9) == 1
    assert d(cap=0) == 1                                                   # a receive buffer holds at least one row
    assert d(x=None) == 2
    assert rf_lib.rf_moe_ep_layout(p16, 0, 3, 8, 64, p16, p16, None) == 1      # 8 experts over 3 ranks
    assert rf_lib.rf_moe_ep_layout(p16, 0, 2, 8, 0, p16, p16, None) == 1       # capacity < 1


# (refused before any device work; where there is a GPU, nothing stands behind these addresses)
no_gpu = pytest.mark.skipif(torch.cuda.is_available(), reason="addresses without memory behind them")

MISALIGNED = 3
A = 0x7000000                # aligned for everything

# entry -> argument list, {argument position: its alignment}
STAGE_ENTRIES = {
    "rf_moe_topk": [([A, 4, 256, 8, A, A, A, None], {0: 16, 4: 4, 5: 2, 6: 4}),
                    ([A, 4, 128, 8, A, A, A, None], {0: 2})],
    "rf_moe_permute": [([A, A, A, 4, 32, 4, A, A, A, A, A, A, None],
                        {0: 4, 1: 4, 2: 2, 6: 4, 7: 4, 8: 4, 9: 4, 10: 2, 11: 4})],
    "rf_moe_gather_rows": [([A, A, 4, 8, 64, A, None], {0: 16, 1: 4, 5: 16})],
    "rf_moe_router_gemm": [([A, A, A, 4, 72, 64, A, None], {0: 16, 1: 16, 2: 4, 6: 16}),
                           ([A, A, A, 4, 32, 64, A, None], {6: 2}), ([A, A, A, 4, 70, 64, A, None], {6: 2})],
    "rf_moe_combine": [([A, A, A, A, 4, 4, 64, A, None], {0: 16, 1: 16, 2: 4, 3: 2, 7: 16})],
    "rf_moe_add_rows": [([A, A, 4, 64, None], {0: 16, 1: 16})],
    "rf_moe_ep_dispatch": [([A, A, A, A, A, 64, 256, 128, 8, 0, 2, 512, (ctypes.c_void_p * 8)(*[A] * 8), None, A, A, A, None],
                            {0: 16, 1: 4, 2: 4, 3: 4, 4: 4, 14: 4, 15: 4, 16: 16})],
    "rf_moe_ep_combine": [([(ctypes.c_void_p * 8)(*[A] * 8), A, A, A, A, A, 4, 4, 64, 2, A, None],
                           {1: 16, 2: 4, 3: 2, 4: 4, 5: 4, 10: 16})],
}


@no_gpu
@pytest.mark.parametrize("entry", STAGE_ENTRIES)
def test_moe_stage_entries_refuse_addresses_that_their_kernels_cannot_take(rf_lib, entry):
    """Half the alignment is refused with a status.  The whole of it is not (the call then fails for want of a device)."""
    fn = getattr(rf_lib, entry)
    for args, aligned in STAGE_ENTRIES[entry]:
        for i, a in aligned.items():
            bad, good = list(args), list(args)
            bad[i], good[i] = A + a // 2, A + a
            assert fn(*bad) == MISALIGNED, (i, a)
            assert fn(*good) not in (0, MISALIGNED), (i, a)


def _layer(n_experts, **fields):
    """A layer's argument block, every address aligned but those given, and what keeps its arrays alive."""
    raw = _lib.MoEInputRaw()
    raw.params = _lib.InputParams(1, 8, 64, 64, n_experts, 2, 1, 0)
    for name in _lib._MOE_PTR_FIELDS:
        setattr(raw, name, fields.get(name, A))
    arrays = {}
    for name in ("expert_weight_gate", "expert_weight_up", "expert_weight_down"):
        arrays[name] = (ctypes.c_void_p * n_experts)(*[A] * (n_experts - 1), fields.get(name, A))
        setattr(raw, name, ctypes.cast(arrays[name], ctypes.POINTER(ctypes.c_void_p)))
    return raw, arrays


@no_gpu
@pytest.mark.parametrize("field,align", [
    ("input_seq", 16), ("expert_weight_gate", 16), ("expert_weight_up", 16), ("expert_weight_down", 16),
    ("shared_expert_weight_gate", 16), ("shared_expert_weight_up", 16), ("shared_expert_weight_down", 16),
    ("expanded_seq_input", 16), ("expanded_fc1_output", 16), ("expanded_fc2_output", 16), ("shared_fc1_output", 16),
    ("shared_fc2_output", 16), ("final_output", 16), ("seq_experts_index", 4), ("source_rows", 4), ("permuted_experts", 4),
    ("permuted_rows", 4), ("first_token_offset", 4), ("rev_permuted_rows", 4), ("seq_experts_softmax", 2),
    ("expanded_seq_softmax", 2)])
def test_moe_layer_refuses_misaligned_addresses_before_it_enqueues_anything(rf_lib, field, align):
    for off, refused in ((align // 2, True), (align, False)):
        raw, keep = _layer(32, **{field: A + off})
        for st in (rf_lib.run_topk(ctypes.byref(raw), None, None), rf_lib.rf_moe_forward(ctypes.byref(raw), None, None, None)):
            assert (st == MISALIGNED) is refused and st != 0


@no_gpu
def test_moe_layer_takes_logits_and_router_as_their_kernels_read_them(rf_lib):
    def status(fn, n_experts, *bias, **fields):
        raw, keep = _layer(n_experts, **fields)
        return fn(ctypes.byref(raw), *bias, None, None)
    topk, forward = rf_lib.run_topk, rf_lib.rf_moe_forward
    # logits: 16 bytes at a time with 256 experts, written by tile stores from 64 experts on, else by the element
    for E, given, computed in ((256, 16, 16), (128, 2, 16), (64, 2, 16), (32, 2, 2)):
        assert status(topk, E, expert_scores=A + given // 2) == MISALIGNED
        assert status(topk, E, expert_scores=A + given) != MISALIGNED
        assert status(forward, E, None, expert_scores=A + computed // 2) == MISALIGNED
        assert status(forward, E, None, expert_scores=A + computed) != MISALIGNED
    # the router's weight and bias where it runs
    assert status(topk, 32, router_weight=A + 8) != MISALIGNED
    assert status(forward, 32, None, router_weight=A + 8) == MISALIGNED
    assert status(forward, 32, A + 2) == MISALIGNED and status(forward, 32, A + 4) != MISALIGNED


def test_expert_parallel_object_validates_its_configuration(rf_lib):
    """rf_moe_ep_create refuses bad configurations before it touches a device."""
    mk = lambda **kw: _lib.RfMoeEpConfig(*[kw.get(n, v) for n, v in (
        ("n_tokens", 64), ("d_hidden", 128), ("d_expert", 64), ("n_routed_experts", 8), ("n_experts_per_token", 2),
        ("n_shared_experts", 1), ("rank", 0), ("world", 2), ("capacity", 0), ("push_results", 1))])
    out = ctypes.c_void_p()
    create = lambda cfg: rf_lib.rf_moe_ep_create(ctypes.byref(cfg), ctypes.byref(out))
    assert create(mk(world=9)) == 1 and create(mk(rank=2)) == 1
    assert create(mk(n_tokens=0)) == 1 and create(mk(d_hidden=100)) == 1
    assert create(mk(n_routed_experts=6)) == 7            # power of two, divisible by the ranks
    assert create(mk(n_experts_per_token=9)) == 7
    assert create(mk(capacity=-1)) == 1
    assert rf_lib.rf_moe_ep_create(None, ctypes.byref(out)) == 2
    assert rf_lib.rf_moe_ep_forward(None, None, None, None) == 2


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    import pytest
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "nope.so"))
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        _lib.lib()


@pytest.mark.parametrize("without", [
    # no torch at all: the binding as a file of its own
    "sys.modules['torch'] = None; import importlib.util as u; s = u.spec_from_file_location('b', {path!r});"
    " m = u.module_from_spec(s); s.loader.exec_module(m); assert b'sm_100a' in m.lib().rf_version()",
    # a torch built without CUDA: the package
    "import torch; [delattr(torch._C, n) for n in ('_cuda_getDevice', '_cuda_getCurrentRawStream')"
    " if hasattr(torch._C, n)]; import radeonflow_kernels_b200 as p; assert p._lib.lib()",
], ids=["torch", "torch with CUDA"])
def test_binding_loads_without(rf_lib, without):
    code = "import sys; " + without.format(path=_lib.__file__)
    res = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr


def test_an_expert_count_beyond_the_weights_is_refused_without_work(rf_lib):
    """The names of a layer's experts are kept from call to call: a bounded number of layers' worth, and none for a
    configuration whose weights are not there."""
    from radeonflow_kernels_b200 import moe
    known = moe._expert_names.cache_info()
    with pytest.raises(KeyError):
        moe._expert_ptrs({"experts.0.0.weight": None}, 100_000, 0, ctypes.c_void_p)
    assert moe._expert_names.cache_info().misses == known.misses
    assert known.maxsize is not None
