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


def kernels(text):
    """(name, body) of every kernel, and of the device functions that hold a kernel's launch order."""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\((?:[^(){}]|\([^()]*\))*\)\s*\{", text):
        yield m.group(1), _block(text, m.end() - 1)


# embed_kernel is the first of a step and is launched without the attribute; decode attention lets its dependents start at once and is
# followed by launches that wait, or by itself
EARLY = {"embed_kernel", "attn_decode_kernel"}


@pytest.mark.parametrize("name", SOURCES)
def test_dependents_start_only_after_the_wait(name):
    """What a launch beside this one relies on: its inputs are complete once the kernel before it lets it start."""
    seen = 0
    for kernel, body in kernels(_text(name)):
        if kernel in EARLY:
            continue
        at = 0
        for m in re.finditer(r"pdl_launch\(\)", body):
            waits = re.findall(r"pdl_wait\(\)", body[at:m.start()])
            assert waits, f"{kernel} lets its dependents start before its own wait"
            at, seen = m.end(), seen + 1
    if re.search(r"pdl_launch\(\)", _text(name)) and not EARLY & {k for k, _ in kernels(_text(name))}:
        assert seen == len(re.findall(r"pdl_launch\(\)", _text(name)))      # every one of them lies in a kernel that was read


def test_kernels_that_leave_their_wait_out_wait_at_their_end():
    found = 0
    for name in SOURCES:
        text = _text(name)
        if "beside" not in text:
            continue
        for kernel, body in kernels(text):
            if "beside" in body:
                assert re.search(r"if \((?:r\.beside|along) && \(blockIdx\.x[^)]*\) == 0\) pdl_wait\(\);\s*\}\s*$", body), kernel
                found += 1
    assert found == 3


def test_a_recurrence_runs_beside_nothing_but_an_attention():
    from mini_llm_b200 import ops
    with pytest.raises(ops.KernelError, match="company"):
        ops.gated_recurrence(None, None, None, None, None, None, 1e-5, None, None, None, heads=1, beside=True)
    again = []
    ops._with_company(lambda: again.append(ops._scope.beside))
    assert again == [True] and not ops._scope.beside


@pytest.mark.parametrize("name", SOURCES)
def test_what_kernels_of_a_step_write_is_not_read_through_l1(name):
    """The flag that sends plain loads to L2 does not reach cp.async, whose 4- and 8-byte form goes through L1."""
    assert "cp.async.ca" not in _text(name)


@pytest.mark.parametrize("name", SOURCES)
def test_what_kernels_of_a_step_write_is_not_read_through_l1(name):
    """The flag that sends plain loads to L2 does not reach cp.async, whose 4-byte form goes through L1: kernels that use it fence
    behind their wait, before the first copy."""
    text = _text(name)
    users = [(k, b) for k, b in kernels(text) if re.search(r"\bcp4\(", b)]
    assert bool(users) == ("cp.async.ca" in text)
    assert len(re.findall(r"cp\.async\.ca", text)) <= 1              # the one in cp4
    for kernel, body in users:
        m = re.search(r"pdl_wait\(\);\s*pdl_launch\(\);\s*if \(!(?:vec|VEC)\) __threadfence\(\);", body)
        assert m and m.end() < re.search(r"\bcp4\(", body).start(), kernel


def test_plain_loads_go_past_l1():
    """Kernels that start before the last one has written what they read, or that do not wait for it at all, rely on it."""
    from mini_llm_b200.csrc import build
    assert build.NVCC_FLAGS[build.NVCC_FLAGS.index("-dlcm=cg") - 1] == "-Xptxas"
