"""Kernels launched by programmatic dependent launch wait for the kernels before
them with every pointer to memory that other kernels write passed to
``dependent_entry``, so that no access through it can be moved before the wait.
Read from the sources: a missing pointer shows as stale data only in a chain
whose order happens to expose it."""

from pathlib import Path
import re

import pytest

CSRC = Path(__file__).resolve().parent.parent/'pyfr_gb300'/'csrc'


def _balanced(s, i, pair='()'):
    """The text inside the bracket that opens at i, and its end."""
    n, j = 0, i
    while True:
        n += (s[j] == pair[0]) - (s[j] == pair[1])
        if n == 0:
            return s[i + 1:j], j
        j += 1


def _kernels(src):
    """{name: (parameters, body)} of the source's kernels."""
    out = {}
    for m in re.finditer(r'__global__', src):
        t = src[m.end():]
        b = re.match(r'\s*void\s*__launch_bounds__', t)
        i = m.end() + (b.end() if b else 0)
        if b:
            _, i = _balanced(src, src.index('(', i))
        name = re.compile(r'\s*(?:void\s+)?(\w+)\s*\(').search(src, i + 1)
        par, j = _balanced(src, src.index('(', name.start(1)))
        body, _ = _balanced(src, src.index('{', j), '{}')
        out[name[1]] = (par, body)
    return out


@pytest.mark.parametrize('path', sorted(CSRC.glob('*.cu')),
                         ids=lambda p: p.name)
def test_written_pointers_pass_the_wait(path):
    src = re.sub(r'//[^\n]*', '', path.read_text())
    launched = set(re.findall(r'b200::launch\(\s*(\w+)', src))
    for name, (par, body) in _kernels(src).items():
        if name not in launched:
            continue
        m = re.search(r'dependent_entry\(', body)
        assert m, f'{name} does not wait'
        args, _ = _balanced(body, m.end() - 1)
        passed = {a.strip().split('.')[0] for a in args.split(',')}
        written = {p.split()[-1].split('__restrict__')[-1].lstrip('*')
                   for p in par.split(',')
                   if '*' in p and 'const' not in p.split('*')[0]}
        assert written <= passed, (name, written - passed)


def test_tensor_core_epilogue_passes_the_wait():
    """The tensor-core apply's epilogue reads and writes the registers of a
    Runge-Kutta stage by plain accesses: through the pointers that passed the
    wait, and not by the non-coherent path, since the kernel writes them."""
    src = re.sub(r'//[^\n]*', '', (CSRC/'mul_umma.cu').read_text())
    i = src.index('void umma_body(')
    body, _ = _balanced(src, src.index('{', i), '{}')
    args = [_balanced(body, m.end() - 1)[0]
            for m in re.finditer(r'dependent_entry\(', body)]
    for f in ('rk_acc', 'rk_u', 'rk_dtp'):
        assert any(f in a.replace(' ', '').split(',') for a in args), f
        assert len(re.findall(rf'p\.{f}\b', body)) == 1, f
    assert '__ldg(acc' not in body and '__ldg(rk_' not in body
