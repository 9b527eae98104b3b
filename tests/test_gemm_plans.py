"""Tuned-plan table of the FP8 GEMM (the replacement of the reference's dispatch table and tuner,
src/gemm/gemm_launcher.cpp:229-247, tuner/gemm_tuner.py): host logic on CPU, effect on the GPU."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from radeonflow_kernels_b200 import tune

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _get(L, m, n, k):
    bn, s = ctypes.c_int(0), ctypes.c_int(0)
    assert L.rf_fp8_gemm_get_plan(m, n, k, ctypes.byref(bn), ctypes.byref(s)) == 0
    return bn.value, s.value


def test_set_get_remove(rf_lib):
    shape = (1088, 1536, 7168)              # not one of the built-in entries
    model = _get(rf_lib, *shape)
    assert model[0] in (128, 256) and model[1] >= 1
    assert rf_lib.rf_fp8_gemm_set_plan(*shape, 128, 2) == 0
    assert _get(rf_lib, *shape) == (128, 2)
    assert rf_lib.rf_fp8_gemm_set_plan(*shape, 0, 0) == 0          # block_n 0 removes the entry
    assert _get(rf_lib, *shape) == model


def test_invalid_entries_are_rejected(rf_lib):
    assert rf_lib.rf_fp8_gemm_set_plan(1024, 1536, 7168, 100, 1) == 1      # tile width
    assert rf_lib.rf_fp8_gemm_set_plan(1024, 1536, 256, 128, 3) == 1       # more slices than K blocks
    assert rf_lib.rf_fp8_gemm_set_plan(1024, 100, 256, 128, 1) == 1        # n % 64
    assert rf_lib.rf_fp8_gemm_get_plan(1024, 100, 256, None, None) == 1


def test_builtin_table_covers_the_benchmark_shapes(rf_lib):
    for (m, n, k) in tune.BENCHMARK_SHAPES:
        bn, s = _get(rf_lib, m, n, k)
        assert bn in (128, 256, 512) and (1 <= s <= k // 128 or s == tune.STREAM_K)


def test_cost_model_names_the_plans_of_the_table(rf_lib):
    """... but two, where pairs and one-CTA tiles of 256 columns are within 5 % of each other."""
    code = ("from tests.test_gemm_plans import _get; from radeonflow_kernels_b200 import _lib, tune; "
            "print([_get(_lib.lib(), *s) for s in tune.BENCHMARK_SHAPES])")
    res = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         env=dict(os.environ, RF_FP8_GEMM_NO_BUILTIN_PLANS="1"))
    assert res.returncode == 0, res.stderr
    model = eval(res.stdout.strip().splitlines()[-1])
    other = {s: (_get(rf_lib, *s), p) for s, p in zip(tune.BENCHMARK_SHAPES, model) if _get(rf_lib, *s) != p}
    assert other == {(1024, 3072, 1536): ((512, 1), (256, 1)), (6144, 1536, 7168): ((256, 1), (512, 1))}


def _plan_list():
    """Plans of shapes around the lines between one pass, split-K in clusters and split-K through memory."""
    from radeonflow_kernels_b200 import _lib
    return [_get(_lib.lib(), m, n, k) for m in (1, 64, 200, 1025, 3000) for n in (64, 576, 1536, 4160)
            for k in (1024, 2176, 4864, 7168)]


def test_plan_without_a_device(rf_lib):
    """The plan of a B200 where there is none: slices of 128-wide tiles whose clusters fit that chip meet in them."""
    assert _get(rf_lib, 64, 576, 7168) == (128, 8)
    assert _get(rf_lib, 200, 1536, 7168) == (128, 5)
    assert _get(rf_lib, 200, 4160, 4864) == (128, 2)


@pytest.mark.parametrize("m,n,k,plan", [
    # a few rows, a wide output: the second launch costs more than it saves (us, this plan / split through memory)
    (4, 6080, 2176, (128, 1)),       # 7.6 / 9.7 in 3 slices
    (3, 5760, 2048, (128, 1)),       # 7.6 / 9.6 in 4 wide slices
    (50, 6784, 2560, (128, 1)),      # 8.3 / 10.7 in 5 wide slices
    # 128-wide slices beat wide ones of the same rounds
    (50, 4480, 4864, (128, 4)),      # 9.4 / 11.7 in 8 wide slices
    (50, 3904, 6784, (128, 4)),      # 9.9 / 11.9 in 8 wide slices
    # but a split through memory pays where it halves a long K loop, and more slices than two in clusters
    (6000, 64, 4096, (128, 3)),      # 8.9 / 10.3 in 2 slices in clusters
    # stream-K does not pay with fewer tiles than SMs
    (300, 4160, 7168, (128, 1)),     # 18.1 / stream-K 26.6
])
def test_plan_of_shapes_where_the_costs_are_close(rf_lib, m, n, k, plan):
    assert _get(rf_lib, m, n, k) == plan


@pytest.mark.parametrize("m,n,k,plan", [
    (6000, 4608, 7168, (512, 1)),    # several rounds of wide tiles: CTA pairs
    (1619, 4096, 1792, (512, 1)),    # two rounds, also of pairs
    (6232, 2304, 2432, (256, 1)),    # 225 pair tiles on 74 pairs: a round more than the wide tiles need
    (1337, 3008, 1920, (256, 1)),    # one round
    (1280, 4096, 7168, (256, tune.STREAM_K)),     # just over one round, long K
    (3655, 2048, 6144, (512, 1)),    # 1.6 rounds: the second one of pairs costs less than stream-K's fixed part
])
def test_plan_between_wide_tiles_pairs_and_stream_k(rf_lib, m, n, k, plan):
    assert _get(rf_lib, m, n, k) == plan
    assert rf_lib.rf_fp8_gemm_workspace_bytes(m, n, k, 1) == 0


def test_pair_plan_of_the_table_asks_for_no_scratch_in_either_layout(rf_lib):
    """The column-major entry, which has no pair kernel, runs such an entry as one pass of 256-wide tiles."""
    assert _get(rf_lib, 1024, 3072, 1536) == (512, 1)
    assert rf_lib.rf_fp8_gemm_workspace_bytes(1024, 3072, 1536, 0) == 0


@pytest.mark.gpu
def test_plan_is_the_same_with_and_without_a_device(rf_lib):
    code = "from tests.test_gemm_plans import _plan_list; print(_plan_list())"
    res = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert res.returncode == 0, res.stderr
    assert res.stdout.strip().splitlines()[-1] == str(_plan_list())


def test_load_plans_file(rf_lib, tmp_path):
    path = tmp_path / "plans.txt"
    path.write_text("# comment\n2112 640 1024 128 2\n\n2112 704 1024 256 1   # trailing\nnot a line\n2112 768 1024 999 1\n")
    assert rf_lib.rf_fp8_gemm_load_plans(str(path).encode()) == -2         # malformed lines reported ...
    assert _get(rf_lib, 2112, 640, 1024) == (128, 2)                       # ... valid ones loaded
    assert _get(rf_lib, 2112, 704, 1024) == (256, 1)
    assert rf_lib.rf_fp8_gemm_load_plans(str(tmp_path / "missing.txt").encode()) == -1
    good = tmp_path / "good.txt"
    tune.write_plans([(2112, 640, 1024, 256, 1, 9.9)], str(good))
    assert rf_lib.rf_fp8_gemm_load_plans(str(good).encode()) == 1
    assert _get(rf_lib, 2112, 640, 1024) == (256, 1)
    for n in (640, 704):
        rf_lib.rf_fp8_gemm_set_plan(2112, n, 1024, 0, 0)


def test_tuner_candidates():
    c = tune.candidates(1024, 512, 7168)
    assert (128, 1) in c and (256, 1) in c and (128, 4) in c
    # tiles already fill the SMs: no split-K, but the ragged last wave (1344 tiles = 9.08 x 148) makes stream-K a candidate
    assert sorted(set(s for (_, s) in tune.candidates(6144, 7168, 2048))) == [tune.STREAM_K, 1]
    assert all(s == 1 for (_, s) in tune.candidates(128 * 148, 256, 1024))   # whole waves: nothing to share out
    assert all(s == tune.STREAM_K or 7168 // 128 // s >= 2 for (_, s) in c)
    assert (512, 1) in tune.candidates(6144, 4608, 7168, pair=True)
    assert tune.parse_shapes("64x128x256,1024X576x7168") == [(64, 128, 256), (1024, 576, 7168)]


@pytest.mark.gpu
@pytest.mark.parametrize("bn,split", [(128, 1), (128, 3), (256, 1), (256, 2)])
def test_registered_plan_is_used_and_correct(rf_lib, bn, split):
    import torch
    from oracle import fp8_gemm as o
    from radeonflow_kernels_b200 import gemm as G
    from tests.helpers import gemm_device_inputs
    m, n, k = 384, 576, 1024
    a, b, a_s, b_s = o.generate_input(m, n, k, 77, "randn")
    assert rf_lib.rf_fp8_gemm_set_plan(m, n, k, bn, split) == 0
    try:
        assert rf_lib.rf_fp8_gemm_choose_split(m, n, k) == split
        assert rf_lib.rf_fp8_gemm_workspace_bytes(m, n, k, 0) == (split * m * n * 4 if split > 1 else 0)
        da, db, das, dbs = gemm_device_inputs(a, b, a_s, b_s)
        c = torch.empty((m, n), dtype=torch.bfloat16, device="cuda:0")
        G.fp8_mm(da, db, das, dbs, c)
        torch.cuda.synchronize()
        assert G.device_status() == 0
        ok, n_bad, max_err = o.check(c.view(torch.uint16).cpu().numpy(), o.fp8_gemm(a, b, a_s, b_s))
        assert ok, (n_bad, max_err)
    finally:
        rf_lib.rf_fp8_gemm_set_plan(m, n, k, 0, 0)


def test_stream_k_plan_entry(rf_lib):
    """A stream-K table entry is honoured where there is a ragged wave worth sharing out, and degrades to the plain
    pass where there is not (whole waves, or shares shorter than two K blocks)."""
    m, n, k = 1088, 3072, 1536                       # 9 x 12 = 108 tiles of 12 K blocks on 148 SMs
    assert rf_lib.rf_fp8_gemm_set_plan(m, n, k, 256, tune.STREAM_K) == 0
    try:
        assert _get(rf_lib, m, n, k) == (256, tune.STREAM_K)
        assert rf_lib.rf_fp8_gemm_workspace_bytes(m, n, k, 0) == 148 * (128 * 256 * 4 + 8)
        assert rf_lib.rf_fp8_gemm_workspace_bytes(m, n, k, 2) == 2 * m * n * 4       # an explicit split still wins
    finally:
        rf_lib.rf_fp8_gemm_set_plan(m, n, k, 0, 0)
    m, n, k = 384, 576, 1024                         # 15 tiles x 8 K blocks: less than two K blocks per SM
    assert rf_lib.rf_fp8_gemm_set_plan(m, n, k, 128, tune.STREAM_K) == 0
    try:
        assert _get(rf_lib, m, n, k) == (128, 1)
        assert rf_lib.rf_fp8_gemm_workspace_bytes(m, n, k, 0) == 0
    finally:
        rf_lib.rf_fp8_gemm_set_plan(m, n, k, 0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(300, 576, 512), (1024, 320, 256), (129, 64, 128), (2048, 1088, 384)])
def test_short_k_two_slab_configuration_with_ragged_tiles(rf_lib, m, n, k):
    """K <= 512 with the 256-wide tile runs the configuration with two store slabs per warp; N values that leave
    the last tile with one 64-column chunk (or a ragged one) exercise the slab alternation across tiles."""
    import torch
    from oracle import fp8_gemm as o
    from radeonflow_kernels_b200 import gemm as G
    from tests.helpers import canary_intact, canary_output, gemm_device_inputs
    a, b, a_s, b_s = o.generate_input(m, n, k, 5 + m, "randn")
    assert rf_lib.rf_fp8_gemm_set_plan(m, n, k, 256, 1) == 0
    try:
        da, db, das, dbs = gemm_device_inputs(a, b, a_s, b_s)
        full, c = canary_output(m, n)
        for _ in range(2):
            G.fp8_mm(da, db, das, dbs, c)
        torch.cuda.synchronize()
        assert G.device_status() == 0
        assert canary_intact(full, m, n)
        ok, n_bad, max_err = o.check(c.view(torch.uint16).cpu().numpy(), o.fp8_gemm(a, b, a_s, b_s))
        assert ok, (n_bad, max_err)
    finally:
        rf_lib.rf_fp8_gemm_set_plan(m, n, k, 0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(2000, 704, 5504), (304, 576, 1024), (48, 4864, 2176)])
def test_workspace_bytes_serve_the_reference_layout_too(rf_lib, m, n, k):
    """The reference-layout entry may split where the row-major one does not; a caller's workspace of the size that
    rf_fp8_gemm_workspace_bytes names is enough for either."""
    import torch
    from oracle import fp8_gemm as o
    from radeonflow_kernels_b200 import gemm as G
    from tests.helpers import canary_intact, canary_output, gemm_device_inputs
    a, b, a_s, b_s = o.generate_input(m, n, k, 4)
    size = rf_lib.rf_fp8_gemm_workspace_bytes(m, n, k, 0)
    ref = o.fp8_gemm(a, b, a_s, b_s)
    for entry, ops in ((rf_lib.rf_fp8_gemm_colmajor, [np.ascontiguousarray(t.T) for t in (a, b, a_s, b_s)]),
                       (rf_lib.rf_fp8_gemm, [a, b, a_s, b_s])):
        dev = gemm_device_inputs(*ops)
        ws = torch.full((size + 64,), 0x5A, dtype=torch.uint8, device="cuda:0")
        full, c = canary_output(m, n)
        split = (0,) if entry is rf_lib.rf_fp8_gemm else ()
        assert entry(*[t.data_ptr() for t in dev], c.data_ptr(), m, n, k, *split, ws.data_ptr(), size, None) == 0
        torch.cuda.synchronize()
        assert G.device_status() == 0 and canary_intact(full, m, n)
        assert bool((ws[size:] == 0x5A).all())
        ok, n_bad, max_err = o.check(c.view(torch.uint16).cpu().numpy(), ref)
        assert ok, (n_bad, max_err)
