"""Every CTA barrier of the kernels stands where all threads of the CTA reach
it: none inside a branch on the thread's index (undefined in CUDA C++ even
where each side has one of its own)."""
import pathlib
import re

import pytest

SRC = pathlib.Path(__file__).resolve().parent.parent / "walicxe2d_b200" / "csrc"
# __syncthreads and the device functions that hold one for the whole CTA
BARRIER = re.compile(r"__syncthreads|\b(?:leaf_end|bar_init_once|grid_barrier|step_grid_sync|nn_sync|nn_wait)\s*\(|"
                     r"\bwait_tiles_p<(?:U|true)>")
THREAD = re.compile(r"\b(?:tid|gtid|lane|warp|row|lo|threadIdx)\b")


def _end(text, at, pair):
    """Index behind the bracket that closes the one at text[at]."""
    depth = 0
    for k in range(at, len(text)):
        depth += (text[k] == pair[0]) - (text[k] == pair[1])
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced")


def _statement(text, at):
    """End of the statement that begins at text[at] (a block or up to ';')."""
    while text[at].isspace():
        at += 1
    if text[at] == "{":
        return _end(text, at, "{}")
    m = re.match(r"(?:if|for|while)\s*\(", text[at:])
    if m:
        return _statement(text, _end(text, at + m.end() - 1, "()"))
    return text.index(";", at) + 1


def thread_branches(text):
    """The text of every branch (and its else) whose condition names the thread."""
    for m in re.finditer(r"\bif\s*\(", text):
        c = _end(text, m.end() - 1, "()")
        if not THREAD.search(text[m.end():c]):
            continue
        e = _statement(text, c)
        yield text[c:e]
        rest = re.match(r"\s*else\b", text[e:])
        if rest:
            yield text[e:_statement(text, e + rest.end())]


@pytest.mark.parametrize("path", sorted(p.name for p in SRC.glob("*.cu*")))
def test_no_cta_barrier_in_a_thread_dependent_branch(path):
    text = re.sub(r"//[^\n]*", "", (SRC / path).read_text())
    found = [b.strip()[:120] for b in thread_branches(text) if BARRIER.search(b)]
    assert not found, found
