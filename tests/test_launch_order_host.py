"""What a dependent launch may leave out of order, read from the sources: evo_hyena_step fetches its states, and evo_gemm_smallm its weights, ahead of their waits, so that a kernel between
them and the one that wrote those orders the two only if it lets its successor start behind its own wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "evo_b200", "csrc")
# launched dependent at every level of evo_set_pdl but 0, by the file that launches them
DEPENDENT = {
    "gemm_tcgen05.cu": {"gemm_tcgen05_kernel"}, "elementwise.cu": {"rmsnorm_row_kernel<false>"}, "attention_pp.cu": {"attn_pp_kernel"}, "window_attention_tc.cu": {"window_attn_tc_kernel"},
    "branch_ops.cu": {"sum_norm_kernel", "sum_norm_row_kernel", "conv_act4_kernel", "conv_act_kernel", "conv_carry_kernel"},
    "delta_block.cu": {"delta_prepare_kernel", "delta_scan_kernel", "delta_single_kernel"},
    "hyena.cu": {"hyena_tc_constants_kernel", "hyena_tc_kernel", "hyena_scan_ms_kernel"},
}
WAIT, START = r"pdl_wait\(\)|griddepcontrol\.wait", r"pdl_launch_dependents\(\)|griddepcontrol\.launch_dependents"


def _text(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def _bodies():
    out = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        s = _text(path)
        for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?:[^()]|\([^()]*\))*\)\s*\{", s):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(s[i], 0)
                i += 1
            if m.group(1) != "__launch_bounds__":
                out[m.group(1)] = s[m.end():i]
    return out


@pytest.mark.parametrize("file,name", [(f, n) for f, names in DEPENDENT.items() for n in sorted(names)])
def test_dependent_kernels_start_their_successor_behind_their_wait(file, name):
    body = _bodies()[name.split("<")[0]]
    if "pdl_enter<" in body:                                 # <true>: the successor first; <false>: the wait first
        assert name.endswith("<false>")
        body = body.replace("pdl_enter<STEP>()", "pdl_wait(); pdl_launch_dependents()")
    wait, start = re.search(WAIT, body), re.search(START, body)
    assert wait is not None, name
    assert start is None or start.start() > wait.start(), name


def test_every_dependent_launch_is_listed():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        s, file = _text(path), os.path.basename(path)
        names = {m.group(1) + (m.group(2) if m.group(2) in ("<true>", "<false>") and m.group(1) == "rmsnorm_row_kernel" else "")
                 for call in re.findall(r"(?<!inline cudaError_t )launch_dependent\(([^;]*?), dim3", s) for m in re.finditer(r"(\w+_kernel)(<\w+>)?", call)}
        names |= set(re.findall(r"launch_after\([^;]*?(\w+_kernel)", s))
        assert names <= DEPENDENT.get(file, set()), (file, names)
        if "ProgrammaticStreamSerialization" in s:
            assert file in DEPENDENT or file == "gemm_smallm.cu", file


def test_tmem_is_held_before_a_successor_may_ask_for_some():
    """A successor that takes the TMEM which a CTA of the kernel in front still asks for, and then waits for that kernel, would wait for good."""
    found = 0
    for name, body in _bodies().items():
        alloc, start = body.find("tmem_alloc<"), re.search(START, body)
        if alloc >= 0 and start is not None:
            found += 1
            barrier = body.find("__syncthreads()", alloc)
            assert 0 <= barrier < start.start(), name
    assert found == 2                                        # gemm_smallm_kernel, gemm_tcgen05_kernel


def test_the_first_launch_of_a_decode_step_is_ordinary():
    """evo_embed_norm is the launch that waits for everything of the step in front."""
    s = _text(os.path.join(CSRC, "elementwise.cu"))
    entry = s[s.index("int evo_embed_norm("):]
    entry = entry[:entry.index("\n}")]
    assert "embed_norm_kernel<long long><<<" in entry and "launch_pdl" not in entry and "launch_dependent" not in entry


def test_level_zero_reaches_every_dependent_launch():
    """evo_set_pdl(0) is off for each launch that carries the attribute."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        s = _text(path)
        for m in re.finditer(r"ProgrammaticStreamSerialization;", s):
            start, end = s.rfind("\n}", 0, m.start()), s.find("\n}", m.start())        # the function around it
            assert re.search(r"pdl_off\(\)|pdl_level\(\) (==|>=) 1", s[start:end]), (os.path.basename(path), s.count("\n", 0, m.start()) + 1)
