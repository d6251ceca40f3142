"""A named barrier inside a loop counts the same warps every time: one that leaves the
loop early, when a bounded wait of its own has run out, would leave the others at the
barrier for good.  So no such loop of the sources has a way out but its count."""
import re

import pytest

from conftest import ROOT

SOURCES = sorted((ROOT / "mocca_gb300" / "csrc").glob("*.cu"))
LOOP = re.compile(r"\bfor \(")


def _close(text, i, pair):
    depth, j = 0, i
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return j


def _loops(text):
    """(header, body) of the for loops with a body in braces."""
    for m in LOOP.finditer(text):
        end = _close(text, m.end() - 1, "()")
        body = re.match(r"\s*\{", text[end:])
        if body:
            start = end + body.end() - 1
            yield text[m.end() - 1:end], text[start:_close(text, start, "{}")]


def _own(body):
    """The loop's body without the loops inside it."""
    for _, inner in _loops(body[1:]):
        body = body.replace(inner, "")
    return body


def _with_barrier():
    for path in SOURCES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for header, body in _loops(text):
            if re.search(r"bar\.sync [1-9]", _own(body)):
                yield pytest.param(header, _own(body), id=f"{path.stem}-{header[:40]}")


@pytest.mark.parametrize("header,body", list(_with_barrier()))
def test_no_way_out(header, body):
    assert "ok" not in re.findall(r"\w+", header)
    assert not re.search(r"\b(?:break|return)\b", body)


def test_found():
    assert len(list(_with_barrier())) == 2
