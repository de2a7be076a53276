"""The kernels of a step are programmatic dependent launches: one may be resident while the one in front of it still
writes what it will read. Read from the sources, as no run shows it: such a kernel waits, its wait clobbers memory, and
what a kernel in front may have written is never read through the non-coherent path (which the wait does not order)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "trixilw.jl_b200", "csrc")

# what the host uploads and no kernel writes, by the names under which the kernels read it
UPLOADED = set("""
    metrics inv_jac inv_jac_node unorm mortar_ij levels now wall w np sf xe xn
    nbr cnbr left right xl xr yl yr lower upper large large_side small1 small2 code mortar_faces
    elem element face faces kind index direction bidx boundary wall_kind p_elem s_elem slot inst atb
""".split())


def sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, f)) as fh:
                out[f] = re.sub(r"//.*", "", fh.read())
    return out


def closing(text, at):
    """The index past the bracket that closes the one at `at`."""
    depth = 0
    for k in range(at, len(text)):
        depth += text[k] in "({["
        depth -= text[k] in ")}]"
        if depth == 0:
            return k + 1
    raise AssertionError("open bracket")


def kernels(text):
    """(name, parameters, body, start, end) of every kernel in a source"""
    for m in re.finditer(r"__global__", text):
        k = text.index("(", m.end())
        if "__launch_bounds__" in text[m.end():k]:
            k = text.index("(", closing(text, k))
        e = closing(text, k)
        b = text.index("{", e)
        yield re.findall(r"(\w+)\s*$", text[:k])[0], text[k:e], text[b:closing(text, b)], m.start(), closing(text, b)


def dependent_names():
    names = set()
    for text in sources().values():
        names |= set(re.findall(r"launch_dependent\([^;]*?,\s*(\w+_kernel)\b", text))
    return names


def dependent_kernels():
    """{name: (parameters, body)} of every kernel that launch_dependent launches"""
    names = dependent_names()
    found = {n: (params, body) for text in sources().values() for n, params, body, _, _ in kernels(text) if n in names}
    assert found.keys() == names and len(names) >= 14
    return found


def test_dependent_kernels_wait():
    for name, (_, body) in dependent_kernels().items():
        wait = body.find("wait_for_previous();")
        assert wait >= 0, name
        for access in (r"\bload\w*\(", r"__ldg\(", r"\batomic\w+\(", r"\*a\.", r"prefetch_next"):
            m = re.search(access, body)
            assert m is None or m.start() > wait, (name, access)


def test_wait_and_coherent_loads_are_ordered():
    text = sources()["tlw_device.cuh"]
    assert re.search(r'asm volatile\("griddepcontrol\.wait;" ::: "memory"\)', text)
    b = text.index("{", text.index("void load4w("))
    assert re.match(r'\{\s*asm volatile\("ld\.global\.v4\.f64 [^;]*;"[^;]*: "memory"\);', text[b:closing(text, b)], re.S)
    b = text.index("{", text.index("void load4("))
    assert "__ldg" not in text[b:closing(text, b)]


@pytest.mark.parametrize("name", [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cuh")])
def test_non_coherent_loads_read_uploaded_data_only(name):
    text = sources()[name]
    # (kernels that are only launched the ordinary way start after everything in front of them has ended)
    for n, _, _, start, end in reversed(list(kernels(text))):
        if n not in dependent_names():
            text = text[:start] + text[end:]
    for m in re.finditer(r"\b(__ldg|load4_const|load4w_const)\(", text):
        arg = text[m.end():closing(text, m.end() - 1) - 1]
        if "const double" in arg and "reinterpret" not in arg or arg.startswith("reinterpret_cast<const double2*>(p)"):
            continue   # the loaders themselves
        arg = re.sub(r"reinterpret_cast<[^>]*>\(", "", arg)
        root = re.match(r"\s*(?:\w+\.)?(\w+)", arg).group(1)
        assert root in UPLOADED, (name, m.group(0) + arg)
    assert ".nc." not in text.replace(NC_LOADER, "")


# the only inline load of the non-coherent path
NC_LOADER = 'asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3]) : "l"(p));'


def test_loader_of_the_non_coherent_path_is_the_const_one():
    text = sources()["tlw_device.cuh"]
    b = text.index("{", text.index("void load4w_const("))
    assert NC_LOADER in text[b:closing(text, b)]


def test_restrict_parameters_of_dependent_kernels():
    """const __restrict__ lets the compiler take the non-coherent path by itself."""
    for name, (params, _) in dependent_kernels().items():
        for p in re.findall(r"const \w+\* __restrict__ (\w+)", params):
            assert p in UPLOADED, (name, p)
