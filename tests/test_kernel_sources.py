"""What the kernels' sources have to keep to and no run can show: rules whose violation is a race or a hang that a machine
may never exhibit.  Read as text; no GPU."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "dl_templates_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def body_at(text, start):
    """The brace-balanced block that opens at or after `start`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[start:j + 1]
    raise AssertionError("unbalanced braces")


def kernels():
    """(name, signature and body) of every __global__ function."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cuh", ".cu")):
            text = source(f)
            for m in re.finditer(r"__global__\s+void", text):
                block = body_at(text, m.start())
                yield re.search(r"(\w+)\s*\((?!\s*\w+\s*[,)]\s*\w+\s*\()", block[block.index("__launch_bounds__") + 18:]).group(1), block


def test_early_started_kernels_read_nothing_through_the_read_only_path():
    """A kernel that is started before its predecessor has finished (pdl_wait) is resident while its inputs are still being
    written: no __ldg (the read-only path wants data that nobody writes while the kernel lives) and no __restrict__ (which the
    compiler may turn into that path, or take as leave to move a load above the wait)."""
    early = [(n, b) for n, b in kernels() if "pdl_wait" in b]
    assert len(early) >= 7
    for name, block in early:
        assert "__ldg" not in block and "__restrict__" not in block and "ld.global.nc" not in block, name
    for helper in ("swa_tc_strip.cuh", "swa_simt_tile.cuh"):          # what those kernels are made of
        assert "__ldg" not in source(helper) and "__restrict__" not in source(helper), helper


def test_a_warp_never_branches_on_one_lanes_view_of_a_barrier():
    """Lanes that test a barrier while its phase completes may see different answers.  A warp that walks a ring together votes on
    the answer: every test or wait in the strip kernels stands inside a warp vote."""
    seen = 0
    for f in ("swa_tc_strip.cuh", "swa_tc_fwd2.cuh", "swa_tc_bwd2.cuh"):
        text = re.sub(r"\s+", " ", source(f))
        for m in re.finditer(r"\b(mbar_test|mbar_wait_polls|mbar_try_wait\w*|mbar_wait)\b", text):
            assert text[:m.start()].rstrip().endswith("__all_sync(0xffffffffu,"), (f, text[m.start() - 80:m.end() + 40])
            seen += 1
    assert seen >= 6


def test_waits_give_up_after_about_a_second():
    """Every bounded wait counts polls that failed.  A failed mbarrier.try_wait takes 1.98 us (3.98 us with a 100 ns hint; a
    test_wait and a short sleep 64 ns), measured: the budgets come to half a second to a second and a half."""
    text = source("umma.cuh") + source("swa_tc_strip.cuh")
    polls = {n: 1 << int(e) for n, e in re.findall(r"\b(k(?:Spin|Park|Load)Polls) = 1u << (\d+)", text)}
    assert set(polls) == {"kSpinPolls", "kParkPolls", "kLoadPolls"}
    for name, ns in (("kSpinPolls", 1980), ("kParkPolls", 3980), ("kLoadPolls", 64)):
        assert 0.5 <= polls[name] * ns * 1e-9 <= 1.5, name
    for f in ("umma.cuh", "swa_tc_strip.cuh", "swa_tc_fwd2.cuh", "swa_tc_bwd2.cuh"):          # ... and no wait has a budget of its own
        assert not re.search(r"(?<!Polls = )1u? << 2\d", source(f)), f
