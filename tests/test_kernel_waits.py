"""Named barriers have no limit: a warp that leaves a loop because one of its bounded mbarrier waits ran out must not leave
others behind at a named barrier of that loop.  Read from the kernels' sources (a wait that runs out cannot be provoked
without holding up a GPU): a loop with a named barrier does not end on `ok`, and where it can be left by `break`, the
barriers that are still to come follow at once, without work between them."""
import re

import pytest

from tests.conftest import ROOT

SOURCES = sorted((ROOT / "joshua_b200" / "csrc").glob("*.cu*"))


def block_end(text, at):
    """The end of the brace block, or of the single statement, that begins at or behind `at`."""
    while text[at].isspace():
        at += 1
    if text[at] != "{":
        return text.index(";", at) + 1
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced braces")


def loops(text):
    """(line, condition, body, what follows) of every loop."""
    for m in re.finditer(r"\b(?:for|while) \(", text):
        depth, i = 1, m.end()
        while depth:
            depth += (text[i] == "(") - (text[i] == ")")
            i += 1
        end = block_end(text, i)
        yield text.count("\n", 0, m.start()) + 1, text[m.end():i - 1], text[i:end], text[end:]


def own_breaks(body):
    """The body without its inner loops, whose breaks are their own."""
    for _, _, inner, _ in loops(body):
        body = body.replace(inner, "")
    return re.search(r"\bbreak;", body)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_a_failed_wait_leaves_nobody_at_a_named_barrier(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    lambdas = {m.group(1): text[m.end() - 1:block_end(text, m.end() - 1)]
               for m in re.finditer(r"auto (\w+) = \[&?[^\]]*\][^{;]*\{", text)}
    meeting = {"bar.sync", "__syncthreads"}
    grown = True
    while grown:  # lambdas that come to a barrier, through others too
        more = {name + "(" for name, body in lambdas.items() if any(b in body for b in meeting)} - meeting
        grown, meeting = bool(more), meeting | more
    for line, condition, body, behind in loops(text):
        held = [b for b in meeting if re.search(r"(?<![\w])" + re.escape(b), body)]
        if held:
            assert not re.search(r"(?<![\w!])ok\b", condition), f"{path.name}:{line}: ends on `ok` and comes to {held}"
        if held and own_breaks(body):
            rest = re.match(r"\s*for \(; [^;]*; [^)]*\) (\w+\()\);", behind)
            assert rest and rest.group(1) in meeting, f"{path.name}:{line}: left by break, comes to {held}"


def test_an_entry_without_a_context_may_have_no_status_flag():
    """The prompt attention takes no context: its flag is NULL until a context exists on the device, so every store through it
    is guarded."""
    text = (ROOT / "joshua_b200" / "csrc" / "attention_prefill.cu").read_text()
    stores = [line for line in text.splitlines() if "volatile int*>(error_flag) = 1" in line]
    assert len(stores) == 2 and all("&& error_flag)" in line for line in stores)
