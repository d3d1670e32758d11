"""A thread block leaves a kernel with none of its bulk copies on the way:
shared memory may have a new owner when they land.  Read from the source: no
`return` of a kernel lies where bytes are expected on a barrier that has not
been waited for, loops taken to run twice.  (A return because the wait itself
gave up is the wait's own affair: it waits a second time.)"""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "mpk_gb300", "csrc")


def _block(text, at):
    """The braces that open at or after `at`: (start, end) of what they hold."""
    i = text.index("{", at)
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if depth == 0:
            return i + 1, j
    raise AssertionError("unbalanced braces")


def _kernels(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"__global__\s+void[^;{]*?(\w+_kernel)\s*\(", text):
        a, z = _block(text, m.end())
        body = text[a:z]
        while True:  # bodies of lambdas are not part of the flow
            q = re.search(r"=\s*\[[&=]?\]\s*(\([^()]*(\([^()]*\))*[^()]*\))?\s*(->[^{]*)?\{", body)
            if not q:
                break
            s, e = _block(body, q.end() - 1)
            body = body[:q.start()] + "= 0" + body[e + 1:]
        yield m.group(1), body


def _twice(text):
    """Loops written out to run twice."""
    out = ""
    for m in iter(lambda: re.search(r"\b(for|while)\s*\([^{;]*(;[^{;]*;[^{;]*)?\)\s*\{", text), None):
        a, z = _block(text, m.end() - 1)
        out += text[:m.start()] + 2 * ("{" + _twice(text[a:z]) + "}")
        text = text[z + 1:]
    return out + text


def _leaves_early(body):
    """The returns with expected bytes outstanding."""
    out, pending = set(), set()
    text = _twice(body)
    for m in re.finditer(r"mbar_expect\(&(\w+)|tr_wait\(&(\w+)|\breturn\b", text):
        if m.group(1):
            pending.add(m.group(1))
        elif m.group(2):
            pending.discard(m.group(2))
        else:
            line = text[max(text.rfind(c, 0, m.start()) for c in ";{}") + 1:m.start()]
            if pending and "!tr_wait(" not in line:
                out.add(" ".join((line + text[m.start():text.index(";", m.start())]).split()))
    return out


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
KERNELS = [(f, k, b) for f in FILES for k, b in _kernels(f)]


def test_finds_the_kernels_with_bulk_copies():
    with_copies = {k for _, k, b in KERNELS if "mbar_expect(" in b}
    assert with_copies >= {"diag_kernel", "batch_pack_kernel", "tiles_reg_kernel"}


@pytest.mark.parametrize("f,k,body", KERNELS, ids=[f"{f}-{k}" for f, k, _ in KERNELS])
def test_no_return_with_copies_on_the_way(f, k, body):
    assert not _leaves_early(body)


@pytest.mark.parametrize("f,k,body", KERNELS, ids=[f"{f}-{k}" for f, k, _ in KERNELS])
def test_flags_are_released(f, k, body):
    """Words that other blocks poll with acquire loads are never stored plainly."""
    assert not re.search(r"\bflags\s*\[[^;]*?\]\s*=[^=]", body)


def test_the_check_sees_an_early_return():
    assert _leaves_early("mbar_expect(&b, 16); if (gave_up) return; tr_wait(&b, 0);")
    assert _leaves_early("for (;;) { if (gave_up) { g(); return; } tr_wait(&b, 0); f(); mbar_expect(&b, 16); }")
    assert not _leaves_early("mbar_expect(&b, 16); if (gave_up) { tr_wait(&b, 0); return; } tr_wait(&b, 0); return;")
