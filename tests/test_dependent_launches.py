"""Kernels launched as programmatic dependents (launch.cuh) read what the iteration writes by
coherent loads: they are resident while their predecessors still write it, and a non-coherent load (__ldg, or
a const __restrict__ pointer) is defined only for data that nobody writes while the kernel lives.
Read from the sources, since a violation need not show in a result."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "meltpooldg_b200",
                    "csrc")
FIXED = {"D"}  # the diagonal: not written during a solve


def sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC))}


def dependent_kernels(src):
    names = set()
    for f, text in src.items():
        if f == "launch.cuh":
            continue
        # directly, or by launch_persistent with its `dependent` argument
        launches = r"launch_dependent\(\s*(\w+)|launch_persistent\(\w+,\s*(\w+)[^;]*?\bdependent\b"
        for m in re.finditer(launches, text):
            name = m.group(1) or m.group(2)
            if name == "kernel":  # launch_persistent itself
                continue
            if not name.startswith("k_"):  # a local: auto k = k_name<...>
                name = re.findall(r"auto %s = (k_\w+)" % name, text[:m.start()])[-1]
            names.add(name)
    return names


def kernel(src, name):
    """(parameters, body) of a kernel's definition."""
    for text in src.values():
        m = re.search(r"__global__[^;{]*?\b%s\(([^)]*)\)\s*\{(.*?)\n\}" % name, text, re.S)
        if m:
            return m.groups()
    raise AssertionError(name)


def test_dependents_read_live_vectors_by_coherent_loads():
    src = sources()
    names = dependent_kernels(src)
    assert names == {"k_vmult2", "k_amr_apply", "k_cg_update_xr", "k_cg_update_p",
                     "k_amr_cg_update", "k_amr_cg_direction"}
    for name in names:
        params, body = kernel(src, name)
        restrict = re.findall(r"__restrict__\s*(\w+)", params)
        assert set(restrict) <= FIXED, (name, restrict)
        wait = body.index("wait_for_predecessor()")
        assert "a.src" not in body[:wait] and "[i]" not in body[:wait], name
        # the operand of an operator kernel
        assert not re.search(r"__ldg\(\s*a\.src", body), name
        for m in re.finditer(r"gather_column<n>\(a\.src, base", body):
            # the FP32 instances', which are not launched as dependents
            assert re.search(r"gather_live<n>\(a\.src[^;]*;\s*\}?\s*else\s*\{?\s*$",
                             body[:m.start()]), name
        if name == "k_vmult2":
            assert len(re.findall(r"gather_live<n>\(a\.src", body)) == 2
    for f in ("cell_args.cuh", "amr_cells.cuh"):
        assert not re.search(r"__restrict__\s+src;", src[f]), f
