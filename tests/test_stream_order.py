"""Kernels read what was copied before them: a copy or memset on the legacy default stream (from
pageable memory it may return before it has landed) is ordered before a kernel on another stream
only by a synchronisation.  Checked on the source, because a lost race cannot be provoked."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "pbh_b200" / "csrc"
LEGACY = re.compile(r"\b(cudaMemcpy|cudaMemset|cudaMemcpyToSymbol)\s*\(")
SYNC = re.compile(r"\bcuda(Device|Stream)Synchronize\s*\(")


def body(file: str, head: str) -> str:
    """The function whose definition starts with `head`, without comments."""
    text = re.sub(r"//[^\n]*", "", (CSRC / file).read_text())
    start = text.index("{", text.index(head))
    depth = 0
    for k in range(start, len(text)):
        depth += (text[k] == "{") - (text[k] == "}")
        if depth == 0:
            return text[start:k + 1]
    raise AssertionError(head)


def unordered(text: str, upto: int):
    """The legacy-stream calls in text[:upto] after the last synchronisation there."""
    syncs = [m.end() for m in SYNC.finditer(text, 0, upto)]
    first = syncs[-1] if syncs else 0
    out = []
    for m in LEGACY.finditer(text, first, upto):
        depth, k = 1, m.end()
        while depth:
            depth += (text[k] == "(") - (text[k] == ")")
            k += 1
        out.append(text[m.end():k - 1])
    return out


def test_the_kernel_of_the_engine_s_creation_reads_finished_tables():
    text = body("engine.cu", "int engine_init(")
    launches = list(re.finditer(r"\blaunch_\w+\s*\(([^;]*)\);", text))
    assert launches
    for m in launches:
        read = re.findall(r"E->d_\w+", m.group(1))
        late = [c for c in unordered(text, m.start()) if any(re.match(re.escape(r) + r"\s*,", c) for r in read)]
        assert not late, late


def test_the_counts_kernels_start_from_cleared_statistics():
    text = body("engine.cu", "int pm_get_counts(")
    at = text.index("launch_deposit(")
    assert "max_fix" in text[:at] and not unordered(text, at)


@pytest.mark.parametrize("file,head", [
    ("native_fft.cu", "int fft_native_init("),   # the twiddle table, read by the first transform on any stream
    ("ic.cu", "int ic_work("),                   # the rms kernel's ticket, counted on the caller's stream
])
def test_set_up_is_complete_when_it_returns(file, head):
    text = body(file, head)
    assert LEGACY.search(text) and not unordered(text, len(text))
