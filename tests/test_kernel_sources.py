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


def test_a_wait_that_gave_up_ends_every_loop_around_it():
    """In the strip kernels a wait polls for about a second whether or not one before it gave up.  A loop that waits, itself or in one
    inside it, is therefore left once `ok` is false: else a warp would give up once per work item.  (Not the loops over the slots of a
    block, four rounds at most, nor the forward kernel's second look at a row, which ends with `if (exact) break`.)"""
    wait = re.compile(r"\b(wait_spin|wait_park|wait|take_ml|load_behind|mbar_wait_polls(?:<\w+>)?)\(")
    left = re.compile(r"if \(!ok(?: \|\| [^;{}]*)?\) (?:break|return);|if \(exact\) break;")
    loops = re.compile(r"\b(?:for|while) \(|\bdo \{")
    seen = 0

    def headers(text):
        for m in loops.finditer(text):
            if m.group().startswith("do"):
                yield m.start(), "", body_at(text, m.start())
                continue
            depth, j = 0, m.end() - 1
            while True:
                depth += {"(": 1, ")": -1}.get(text[j], 0)
                if depth == 0:
                    break
                j += 1
            if text[j + 1:].lstrip().startswith("{"):
                yield m.start(), text[m.end():j], body_at(text, j + 1)

    for f in ("swa_tc_strip.cuh", "swa_tc_fwd2.cuh", "swa_tc_bwd2.cuh"):
        text = re.sub(r"\s+", " ", source(f))
        for at, head, block in headers(text):
            if not wait.search(block) or re.search(r"\w+ &= \w+ - 1$", head.strip()):
                continue
            own = block
            for _, _, inner in headers(block[1:]):
                own = own.replace(inner, "if (!ok) return;" if "if (!ok) return;" in inner else "")
            seen += 1
            assert re.match(r"[^;]*;\s*ok && ", head) or left.search(own), (f, text[at:at + 120])
    assert seen >= 10
