"""A block may write to another one's shared memory only once that block has
started: every kernel of the sources that runs in clusters waits at a cluster
barrier before its first store, arrival or copy to another block."""
import re

import pytest

from conftest import ROOT

SOURCES = sorted((ROOT / "mocca_gb300" / "csrc").glob("*.cu"))
BARRIER = re.compile(r"barrier\.cluster\.wait|\b(?:cluster_barrier|pair_barrier)\(\)")
REMOTE = re.compile(r"st\.shared::cluster|st\.async|shared::cluster\.b64 _|"
                    r"\b(?:put_remote|peer_arrive|store_all|cluster_sum|grid_sum)\(")


def _body(text, start):
    """From the kernel's opening brace to the one that closes it."""
    i = text.index("{", text.index(")", text.index("(", text.index("k_", start))))
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def _cluster_kernels():
    for path in SOURCES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__cluster_dims__", text):
            name = re.search(r"\b(k_\w+)\s*\(", text[m.end():]).group(1)
            yield pytest.param(_body(text, m.end()), id=f"{path.stem}-{name}")


@pytest.mark.parametrize("body", list(_cluster_kernels()))
def test_barrier_before_the_first_store(body):
    remote, barrier = REMOTE.search(body), BARRIER.search(body)
    assert remote is not None and barrier is not None
    assert barrier.start() < remote.start()
