"""Kernels that may start before the one in front of them has drained
(``launch_chained``, csrc/common.cuh) wait first and read global memory with
coherent loads only: the compiler may move a non-coherent one (``__ldg``, a load
through a ``const __restrict__`` pointer) ahead of the wait.  Read from the
sources; needs no GPU."""
import glob
import os
import re

from mnpbem_b200.build import CSRC

SOURCES = {os.path.basename(f): re.sub(r'//[^\n]*', '', open(f).read())
           for f in sorted(glob.glob(os.path.join(CSRC, '*.cu*')))}


def _block(src, i, opening, closing):
    """End of the bracketed text that opens at src[i]."""
    depth = 0
    for j in range(i, len(src)):
        depth += {opening: 1, closing: -1}.get(src[j], 0)
        if depth == 0:
            return j + 1
    raise AssertionError('unbalanced')


def _kernels():
    """name -> list of (file, parameters, body) of every __global__ function."""
    out = {}
    for name, src in SOURCES.items():
        for m in re.finditer(r'__global__\s+void\b', src):
            i = m.end()
            b = re.match(r'\s*__launch_bounds__\s*', src[i:])
            if b:
                i = _block(src, i + b.end(), '(', ')')
            k = re.match(r'\s*(\w+)\s*', src[i:])
            p0 = i + k.end()
            p1 = _block(src, p0, '(', ')')
            b0 = src.index('{', p1)
            out.setdefault(k.group(1), []).append((name, src[p0:p1],
                                                   src[b0:_block(src, b0, '{', '}')]))
    return out


def test_waiting_kernels_use_coherent_loads():
    waiting = [(n, d) for n, ds in _kernels().items() for d in ds if 'grid_wait()' in d[2]]
    assert len(waiting) >= 12
    for n, (f, params, body) in waiting:
        assert '__restrict__' not in params, (f, n)
        assert not re.search(r'__ldg|__ldcs|__ldlu|ld\.global\.nc', body), (f, n)
        # nothing is read before the wait: declarations and named constants only
        head = body[:body.index('grid_wait()')]
        assert not re.search(r'\[[^\]]*\]\s*=|=\s*\*|\bload|\bld\(', head), (f, n)


def test_chained_launches_are_of_waiting_kernels():
    kernels, seen = _kernels(), set()
    for f, src in SOURCES.items():
        for m in re.finditer(r'launch_chained\("[^"]*",\s*(\w+)', src):
            seen.add(m.group(1))
            # skinny.cuh picks one of two instances before the launch
            names = ['kernel', 'mma_kernel'] if m.group(1) == 'f' else [m.group(1)]
            for n in names:
                if f == 'skinny.cuh':
                    defs = [d for d in kernels[n] if d[0] == f]
                else:
                    defs = [d for d in kernels[n] if d[0] == f or len(kernels[n]) == 1]
                assert defs and all('grid_wait()' in d[2] for d in defs), (f, n)
    assert len(seen) >= 10
