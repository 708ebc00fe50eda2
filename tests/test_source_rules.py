"""Rules of the CUDA sources that no launch can show: read from the text, without a GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mini_llm_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _block(text, at):
    """The braces that open at or after ``at``, with what is between them."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced braces")


def once_guards(text):
    """(flag, block) of every `static flag; if (!flag) { ... }` that raises a kernel's limit of shared memory."""
    for m in re.finditer(r"static (?:bool|int) (\w+)(?:\[\d+\])?\s*=", text):
        g = re.compile(r"if \([^;{]*!%s\b[^;{]*\)\s*\{" % m.group(1)).search(text, m.end())
        if g and "cudaFuncSetAttribute" in _block(text, g.end() - 1):
            yield m.group(1), _block(text, g.end() - 1)


@pytest.mark.parametrize("name", SOURCES)
def test_a_first_call_is_marked_done_after_it_is_done(name):
    """A second thread that finds the flag set launches at once, and a call that failed is made again."""
    for flag, block in once_guards(_text(name)):
        written = [m.start() for m in re.finditer(r"(?:&%s\b|\b%s(?:\[\w+\])?\s*=[^=])" % (flag, flag), block)]
        assert written, (name, flag)
        assert min(written) > block.rindex("cudaFuncSetAttribute"), (name, flag)


def test_the_guards_are_found():
    assert sum(len(list(once_guards(_text(n)))) for n in SOURCES) >= 12
