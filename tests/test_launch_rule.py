"""The rule of kernels launched so that they may start early (launch_after in
api.cu), checked on the sources: a load that the compiler may take for one of
constant memory could be moved ahead of the kernel's wait for what came before
it on the stream, so no argument of such a kernel is marked __restrict__ and
none of its own lines uses __ldg; and only a kernel that waits itself is
promised to see what the kernels before it wrote, so the wait is the first
thing that each of them does."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "plasmasim_b200", "csrc")
TEXT = {f: re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def until_closed(text, start, pair):
    """Index behind the bracket that closes the one at `start`."""
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def early_kernels():
    names = set()
    for text in TEXT.values():
        for m in re.finditer(r"launch_after\(c,", text):
            call = text[m.start():until_closed(text, text.index("(", m.start()), "()")]
            names |= set(re.findall(r"\b(\w+_kernel)\b", call))
    return sorted(names)


def definition(name):
    """(arguments, body) of a kernel."""
    for text in TEXT.values():
        m = re.search(r"\b" + name + r"\s*\(", text)
        while m:
            end = until_closed(text, m.end() - 1, "()")
            if re.match(r"\s*\{", text[end:]):
                start = text.index("{", end)
                return text[m.end():end - 1], text[start:until_closed(text, start, "{}")]
            m = re.compile(r"\b" + name + r"\s*\(").search(text, end)
    raise AssertionError(name)


def test_the_kernels_are_found():
    assert {"push_tiled_kernel", "place_fill_kernel", "scan_tile_kernel", "thrust_kernel"} <= set(early_kernels())


@pytest.mark.parametrize("name", early_kernels())
def test_no_load_ahead_of_the_wait(name):
    args, body = definition(name)
    assert "__restrict__" not in args and "__restrict__" not in body and "__ldg" not in body


def test_windows_are_filled_behind_the_wait():
    """fill_win's addresses are known when the kernel starts."""
    text = TEXT["push_tiled.cuh"]
    start = text.index("fill_win(")
    body = text[start:until_closed(text, text.index("{", start), "{}")]
    assert "__ldg" not in body


@pytest.mark.parametrize("name", early_kernels())
def test_waits_first(name):
    _, body = definition(name)
    assert re.match(r"\{\s*after_prior\(\);", body)
