"""Kernels that may start before the kernel ahead of them has finished
(launch_after) read what that kernel is still writing, after a wait. A const
__restrict__ pointer would let the compiler take such data for constant over
the kernel's lifetime and load it through the read-only path, which the wait
does not order: neither these kernels nor the device functions of the same
files that they call may use one."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "fast-general-gpu-sph-framework_gb300" / "csrc"
DEFINITION = re.compile(r"(?:__global__|__device__)[^;{]*?\b(\w+)\s*\((?=[^;]*?\)\s*\{)", re.S)
READ_ONLY = re.compile(r"const\s+[\w\s]+\*\s*(?:const\s+)?__restrict__|__ldg\s*\(")


def code(path):
    """The file without comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def functions(text):
    """name -> texts (signature and body) of the device functions in a file."""
    out = {}
    for m in DEFINITION.finditer(text):
        name = m.group(1)
        if name == "__launch_bounds__":   # the name follows the bounds
            name = re.compile(r"\)\s*(\w+)\s*\(").search(text, m.end()).group(1)
        at = depth = text.index("{", m.end())
        depth = 0
        for k in range(at, len(text)):
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            if depth == 0:
                out.setdefault(name, []).append(text[m.start():k + 1])
                break
    return out


def offenders(texts):
    """Functions reached by dependent launches that promise constant data."""
    funcs = {}
    for t in texts:
        for name, bodies in functions(t).items():
            funcs.setdefault(name, []).extend(bodies)
    todo = {n for n, bodies in funcs.items() if any("chain_wait()" in b for b in bodies)}
    seen = set()
    while todo:
        n = todo.pop()
        seen.add(n)
        for b in funcs[n]:
            todo |= {c for c in re.findall(r"\b(\w+)\s*(?:<[^;()]*>)?\s*\(", b)
                     if c in funcs and c not in seen}
    return seen, sorted(n for n in seen if any(READ_ONLY.search(b) for b in funcs[n]))


def test_dependent_kernels_promise_no_constant_data():
    texts = [code(CSRC / n) for n in ("gsph_internal.h", "split_device.cuh", "grid.cu")]
    seen, bad = offenders(texts)
    assert {"k_cell_scan", "k_scatter", "k_sort_small", "k_sort_big", "cell_model",
            "load_tile_counts"} <= seen
    assert bad == []
    seen, bad = offenders([code(CSRC / n) for n in ("gsph_internal.h", "physics.cu")])
    assert {"k_density_tra", "k_density_tra_rows", "row_range"} <= seen
    assert bad == []


def test_every_dependent_kernel_waits_first():
    for name in ("grid.cu", "physics.cu"):
        text = code(CSRC / name)
        funcs = functions(text)
        launched = set(re.findall(r"launch_after\(\s*(?:motion \? )?(k_\w+)", text))
        launched |= {"k_cell_scan", "k_sort_big"} if name == "grid.cu" else {"k_density_tra"}
        assert launched
        for k in launched:
            for b in funcs[k]:
                first = b[b.index("{") + 1:]
                # (declarations of shared memory do nothing)
                first = re.sub(r"^\s*(?:(?:__shared__|constexpr)[^;]*;\s*)*", "", first)
                assert first.startswith("chain_wait();"), k
