"""Kernels that are launched ahead of their predecessor's end (pdl_wait) read what it wrote: not
through the read-only path, whose loads need data that nothing writes while the kernel lives."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / 'mpdugks_gb300' / 'csrc'
# the D2V16 matrix: written once, when the handle is made
CONSTANT = ('P.iM16',)


def with_headers(path, seen):
    if path in seen or not path.exists():
        return seen
    seen.append(path)
    for name in re.findall(r'#include "([^"]+)"', path.read_text()):
        with_headers(CSRC / name, seen)
    return seen


def early_files():
    out = [p for p in CSRC.glob('*.cu') if any('pdl_wait();' in q.read_text() for q in with_headers(p, []))]
    assert len(out) >= 5
    return out


def test_no_read_only_loads_of_what_a_predecessor_writes():
    found = []
    for path in {q for p in early_files() for q in with_headers(p, [])}:
        text = re.sub(r'//[^\n]*', '', path.read_text())
        for m in re.finditer(r'__ldg\(([^;\n]*)|ld\.global\.nc', text):
            if not (m.group(1) or '').startswith(CONSTANT):
                found.append((path.name, m.group(0)))
    assert not found


def test_early_kernels_take_no_read_only_pointers():
    found = []
    for path in {q for p in early_files() for q in with_headers(p, [])}:
        text = re.sub(r'//[^\n]*', '', path.read_text())
        for m in re.finditer(r'__global__[^{;]*?\b(k_\w+)\(([^{]*?)\)\s*\{([^\n]*\n){1,6}', text):
            if 'pdl_wait();' in m.group(0) and '__restrict__' in m.group(2):
                found.append((path.name, m.group(1)))
    assert not found
