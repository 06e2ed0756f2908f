"""Rules for the kernels' sources that no run on one device can show broken."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mivi_v4_b200", "csrc")


def sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def test_instructions_of_a_whole_warp_are_volatile():
    """An instruction that all lanes of a warp must reach together may not be moved behind a branch that some of them skip, which the
    compiler is free to do with an asm statement that is not volatile."""
    found = [f"{name}: {m.group(1)[:60]}" for name, text in sources()
             for m in re.finditer(r'asm\s*\(\s*"([^"]*)"', text) if ".sync" in m.group(1) or ".aligned" in m.group(1)]
    assert not found, found


def test_shared_memory_is_allowed_on_every_device():
    """A kernel's permission for more shared memory belongs to a device: asked for once in a process, its launches on another device fail.
    (float32 models ran on any device of a process before their kernels needed the permission.)"""
    once = [name for name, text in sources() if re.search(r"static\s+(const\s+)?cudaError_t[^;]*cudaFuncSetAttribute", text)]
    assert not once, once


def test_tensor_memory_is_accessed_by_whole_warps():
    """Loads, stores and the return of tensor memory are .sync.aligned: lanes that come from a branch by row (a row's sink, a row beyond the last) have to
    be together again, which only a __syncwarp right before the instruction assures."""
    found, seen = [], 0
    for name, text in sources():
        for m in re.finditer(r'asm volatile\(\s*"(tcgen05\.(?:ld|st|dealloc)[^"]*)"', text):
            seen += 1
            if not text[:m.start()].rstrip().endswith("__syncwarp();"):
                found.append(f"{name}: {m.group(1)[:60]}")
    assert not found and seen > 10, found


def test_error_codes_name_their_kernel():
    """Every bounded wait's code belongs to one kernel, and the error's text names it; 4 is a guarded index."""
    from mivi_v4_b200.ops.kernels import _error_text
    codes = {}
    for name, text in sources():
        for m in re.finditer(r"\berr, (\d+)\)", text):
            codes.setdefault(int(m.group(1)), set()).add(name)
    assert codes.pop(4) == {"common.cuh"} and len(codes) > 40
    for code, files in codes.items():
        assert len(files) == 1 and f"({min(files)}, code {code})" in _error_text(0, code), (code, files)
        assert "outside its bounds" not in _error_text(0, code)
    assert "outside its bounds" in _error_text(0, 4) and "unknown" in _error_text(0, 999)
