"""The library's own choice of transform per axis length (asg_debug_line_plan)."""
import ctypes as C
import functools
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "angularspectrum_heterogeneous_gb300")


@functools.lru_cache(maxsize=1)
def plans():
    """{n: (direct, variant, n1, n2)} for n = 1 .. 2048."""
    path = os.path.join(PKG, "libasgb300.so")
    if not os.path.exists(path):
        import __graft_entry__ as g
        g.build()
    lib = C.CDLL(path)
    out = {}
    for n in range(1, 2049):
        v = [C.c_int() for _ in range(4)]
        assert lib.asg_debug_line_plan(n, *map(C.byref, v)) == 0, n
        out[n] = tuple(x.value for x in v)
    return out


def compiled_chirps():
    """The convolution lengths (n1, n2) that kernels are compiled for."""
    src = open(os.path.join(PKG, "csrc", "asg_lines.cuh")).read()
    body = re.search(r"#define ASG_CHIRP_SIZES\(F\)((?:.*\\\n)*.*\n)", src).group(1)
    return {tuple(map(int, m)) for m in re.findall(r"F\((\d+), (\d+)\)", body)} | {(64, 64)}


def edge_lengths():
    """Lengths that together run every compiled transform: of each convolution the smallest and
    the largest n, of each radix of a direct variant, as either factor, the smallest n."""
    found = {}
    for n, (direct, variant, n1, n2) in plans().items():
        if direct:
            found.setdefault(("n1", variant, n1), [n])
            found.setdefault(("n2", variant, n2), [n])
        else:
            found.setdefault((n1, n2), [n, n])[1] = n
    return sorted({n for v in found.values() for n in v if n >= 3})
