"""Overlapped launches (programmatic dependent launch) are ordered only if no block of a kernel ends before its wait: a grid whose blocks all left in
front of theirs is complete while the kernel before it still runs, and the next kernel waits for that grid alone.  Read from the sources, so
that it needs no GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mini_inference_engine_b200", "csrc")
WAIT = re.compile(r"\b(?:pdl_wait|pdl_enter|grid_dep_wait)\s*\(\s*\)\s*;")


def _plain(text: str) -> str:
    """The source without comments and strings (replaced by blanks, so that offsets stay); a wait written out becomes a call."""
    text = re.sub(r"asm volatile\(\"griddepcontrol\.wait;\"[^;]*;", lambda m: "pdl_wait();".ljust(len(m.group(0))), text)
    blank = lambda m: re.sub(r"[^\n]", " ", m.group(0))
    return re.sub(r"//[^\n]*|/\*.*?\*/|\"(?:\\.|[^\"\\\n])*\"", blank, text, flags=re.S)


def _matching(text: str, at: int, pair: str) -> int:
    """The index of the bracket that closes the one at ``at``."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced brackets")


def kernels():
    """(file, name, body) of every __global__ function that is defined in the package."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = _plain(open(path).read())
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"(?:__launch_bounds__\s*)|(\w+)\s*(?=\()").search(text, m.end())
            if head.group(0).startswith("__launch_bounds__"):
                close = _matching(text, text.index("(", head.start()), "()")
                head = re.compile(r"(\w+)\s*(?=\()").search(text, close)
            close = _matching(text, text.index("(", head.end(1)), "()")
            begin = re.compile(r"\s*([{;])").match(text, close + 1)
            if begin.group(1) == "{":
                yield os.path.basename(path), head.group(1), text[begin.start(1):_matching(text, begin.start(1), "{}") + 1]


def leaves_before_its_wait(body: str) -> list:
    """Lines of ``return;`` that a block can reach without having waited: not behind a wait of the same block of statements or of one around it.
    (A lambda's return leaves the lambda only.)"""
    waited, left = [False], []
    for m in re.finditer(r"[{}]|\breturn\s*;|" + WAIT.pattern, body):
        token = m.group(0)
        if token == "{":
            waited.append(waited[-1] or re.search(r"\]\s*(?:\([^()]*\))?\s*(?:mutable)?\s*$", body[:m.start()]) is not None)
        elif token == "}":
            waited.pop()
        elif token.startswith("return"):
            if not waited[-1]:
                left.append(body[:m.start()].count("\n"))
        else:
            before = body[:m.start()].rstrip()
            if before[-1] in ";{}":                                    # (a statement of its own, not the arm of an `if`)
                waited[-1] = True
    return left


def test_the_reader_itself():
    assert leaves_before_its_wait("{ if (x) return; pdl_wait(); if (y) return; }") == [0]
    assert leaves_before_its_wait("{ if (x) { pdl_wait(); return; } if (y) return; pdl_wait(); }") == [0]
    assert leaves_before_its_wait("{ if (x) { pdl_wait(); return; } pdl_wait(); { return; } }") == []
    assert leaves_before_its_wait("{ if (x) pdl_wait(); return; }") == [0]
    assert leaves_before_its_wait("{ auto f = [&](int n) { return; }; pdl_wait(); return; }") == []
    assert leaves_before_its_wait(_plain('{ asm volatile("griddepcontrol.wait;" ::: "memory"); return; }')) == []


def test_no_block_leaves_before_its_wait():
    found = {f"{file}: {name}": lines for file, name, body in kernels() if WAIT.search(body) and (lines := leaves_before_its_wait(body))}
    assert not found, found


def test_every_overlapped_kernel_waits():
    """A kernel that is launched with the attribute and never waits would end the chain as well."""
    plainly = set()                                                    # launched with <<< >>>, hence after all that came before
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        plainly |= set(re.findall(r"(\w+)\s*(?:<[^<>;]*>)?\s*<<<", _plain(open(path).read())))
    found = list(kernels())
    assert len(found) > 60
    without = [f"{file}: {name}" for file, name, body in found if name not in plainly and not WAIT.search(body)]
    assert not without, without
