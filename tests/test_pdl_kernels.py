"""Kernels of programmatic dependent launches: no grid ends before the grid ahead of it.  Either no thread
leaves before its wait, or the launch is left out where every block would.  And what the grid ahead may
write is not read as data that is constant for the kernel's life.  Read off the sources (no GPU): what
a kernel does not wait for depends on timing."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lynx_b200", "csrc")


def _kernels():
    """(name, parameters, body) of every kernel that calls pdl_wait(), comments taken out."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as fh:
            src = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\)?\s*)?(\w+)\s*\(([^;{]*?)\)\s*\{", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            if "pdl_wait();" in src[m.end():i]:
                out.append((m.group(1), m.group(2), src[m.end():i]))
    return out


KERNELS = _kernels()


def test_the_kernels_are_found():
    assert {k[0] for k in KERNELS} >= {"direct_step_kernel", "nonorth_mixed_kernel", "nl_atom_kernel"}


# kernels some of whose blocks leave early: where they are launched, and what is asked before
GUARDED = {"nl_atom_kernel": ("nonlocal_launch.cu", "launch_atom_kernel", "if (nl.max_np == 0) return LYNX_OK;")}


@pytest.mark.parametrize("name,params,body", KERNELS, ids=[k[0] for k in KERNELS])
def test_no_grid_leaves_before_the_wait(name, params, body):
    wait = body.index("pdl_wait();")
    early = [m.start() for m in re.finditer(r"\breturn;", body) if m.start() < wait]
    if name not in GUARDED:
        assert not early, f"{name} leaves before pdl_wait()"
        return
    assert len(early) == 1 and "if (np == 0) return;" in body[:wait]
    path, launcher, guard = GUARDED[name]
    with open(os.path.join(CSRC, path)) as fh:
        src = fh.read()
    assert src.count(name + "<") == src.count("go(" + name + "<")  # one launcher
    text = src[src.index("int " + launcher + "("):]
    assert -1 < text.find(guard) < text.index("launch_pdl(")


@pytest.mark.parametrize("name,params,body", KERNELS, ids=[k[0] for k in KERNELS])
def test_no_constant_pointers(name, params, body):
    assert not re.search(r"\bconst\b[^,]*\*\s*__restrict__", params) and "__ldg(" not in body
