"""Kernels whose start may overlap the end of the kernel before them (they begin with pdl_start()) exist while that
kernel still writes.  The read-only load path (__ldg, const __restrict__ arguments) promises data that nobody
writes in a kernel's lifetime, so such kernels, and every device function they call, may use it for links only
(ld_link: link writers end with a wait of the host).  Read from the sources, no GPU needed."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "qkxtm_mpi_b200", "csrc")


def _functions():
    """name -> [(parameters, body)] of every function definition of the CUDA sources."""
    out = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        s = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"\b(\w+)\s*\(", s):
            k, depth = m.end(), 1
            while k < len(s) and depth:
                depth += {"(": 1, ")": -1}.get(s[k], 0)
                k += 1
            tail = re.match(r"\s*(const\s*)?\{", s[k:])
            head = s[max(0, s.rfind(";", 0, m.start()), s.rfind("}", 0, m.start())):m.start()]
            if m.group(1) in ("for", "if", "while", "constexpr") or not tail:
                continue
            if not re.search(r"__(global|device)__", head):
                continue
            b0 = k + tail.end()
            b, depth = b0, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(s[b], 0)
                b += 1
            out.setdefault(m.group(1), []).append((s[m.end():k - 1], s[b0:b]))
    return out


def test_overlapping_kernels_read_written_data_with_plain_loads():
    fn = _functions()
    kernels = [n for n, defs in fn.items() if any("pdl_start()" in b for _, b in defs)]
    assert {"hop_s2_kernel", "k_gauss_step", "k_redot", "k_finalize", "k_cg_finalize", "k_cg_update", "k_axpy_h",
            "k_xpay_h"} <= set(kernels)
    for kernel in kernels:
        for par, body in fn[kernel]:
            assert "__restrict__" not in par, kernel
        seen, todo = set(), [kernel]
        while todo:
            name = todo.pop()
            if name in seen or name == "ld_link":
                continue
            seen.add(name)
            for _, body in fn[name]:
                assert not re.search(r"\b(__ldg|ldc|LdNc)\b|\.load(_raw)?\(", body), (kernel, name)
                for arg in re.findall(r"\bld_link\(\s*(\w+)", body):
                    assert arg in ("ub", "ul"), (kernel, name, arg)  # pointers into the links
                todo += [w for w in re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", body) if w in fn]
        if kernel == "hop_s2_kernel":
            assert {"hop_side_s2", "s2_epilogue", "ld_field"} <= seen  # the walk reaches the loads


def test_kernels_launched_to_overlap_begin_with_the_wait():
    fn = _functions()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for name in re.findall(r"\blaunch_pdl\(c, (\w+)", open(path).read()):
            for _, body in fn[name]:
                first = body.strip().split(";")[0]
                assert first in ("pdl_start()", "if constexpr (PDL) pdl_start()"), name
