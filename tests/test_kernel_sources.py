"""Rules of the kernels that no result shows when they are broken: what they break is an order that the hardware keeps
nearly always.  Checked on the kernels' source text."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "radeonflow_kernels_b200", "csrc")


def _text(path):
    """Source without comments."""
    with open(path) as f:
        s = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", s, flags=re.S)


def _closing(s, start, pair):
    depth = 0
    for i in range(start, len(s)):
        depth += (s[i] == pair[0]) - (s[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced " + pair)


def _kernels():
    """(file, kernel, parameter list, body) of every kernel."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        s = _text(path)
        for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\((?:[^()]|\([^()]*\))*\)\s*)*(\w+)\s*\(", s):
            end = _closing(s, m.end() - 1, "()")
            body = s.index("{", end)
            out.append((os.path.basename(path), m.group(1), s[m.end():end], s[body:_closing(s, body, "{}") + 1]))
    return out


KERNELS = _kernels()
IDS = [f"{f}:{name}" for f, name, _, _ in KERNELS]


def test_every_kernel_is_found():
    n = sum(len(re.findall(r"__global__", _text(p))) for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    assert len(KERNELS) == n and n > 10


@pytest.mark.parametrize("kernel", KERNELS, ids=IDS)
def test_commits_on_stage_barriers_are_waited_for(kernel):
    """A tcgen05.commit that frees a stage arrives on the stage's barrier by itself: the producer waits for the last ones, or
    they could arrive in shared memory that another CTA has taken over."""
    _, _, _, body = kernel
    if re.search(r"umma_commit\w*\(\s*empty_bar", body):
        assert re.search(r"finish_producer\((ok, it|loads_ok, loads), \w+, empty_bar\(0\)", body)


def test_a_scale_slot_is_given_back_by_its_readers():
    """The pair kernel's scale warps rewrite a slot behind a barrier on which the epilogue warps that read it have arrived
    with release semantics; the accumulator's hand-back (relaxed arrive, commit) orders no shared-memory read."""
    body = next(b for _, name, _, b in KERNELS if name == "fp8_gemm_pair_kernel")
    scales, epilogue = body[body.index("warp >= 2"):].split("setmaxnreg.inc", 1)
    assert scales.index("mbar_wait(scale_empty_bar(buf)") < scales.index("st_shared_v4(slot")
    assert "tmem_full_bar(buf), (q" not in scales
    assert epilogue.index("ld_shared_u32(my_scale") < epilogue.index("mbar_arrive(scale_empty_bar(buf))")


def test_dependent_launches_read_nothing_as_constant_data():
    """A kernel that may start before the one in front of it has finished waits for it and then reads what it wrote: with loads
    that the compiler cannot move in front of that wait.  (In files with such kernels, the helpers they call included.)"""
    waiting = [(f, name, params) for f, name, params, body in KERNELS if "griddep_wait()" in body]
    assert len(waiting) >= 8
    for f, name, params in waiting:
        assert not re.search(r"const[^,]*\*\s*__restrict__", params), (f, name)
    for f in {f for f, _, _ in waiting} | {"ptx.cuh", "fp8_tiles.cuh"}:
        assert not re.search(r"__ld(g|cg|ca|cs|lu)\(", _text(os.path.join(CSRC, f))), f


def test_dependent_launches_wait():
    """Files that launch kernels as programmatic dependents: each of their kernels waits, or is launched without."""
    plain = {"sort_count_kernel", "tile_list_kernel"}      # `launch(..., false, ...)`, <<< >>>
    for f, name, _, body in KERNELS:
        if "programmaticStreamSerializationAllowed" in _text(os.path.join(CSRC, f)) and name not in plain:
            assert body.count("griddep_wait()") == 1, (f, name)
    s = _text(os.path.join(CSRC, "moe_route.cu"))
    assert re.search(r"launch\(sort_count_kernel, [^;]*?, stream, false,", s) and "tile_list_kernel<<<" in s
