"""Every entry point that launches, allocates or clears device memory first makes its context's device the
calling thread's (a program may hold contexts on several devices in one thread)."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = os.path.join(ROOT, "optical-pathtracer_b200", "csrc", "owec_api.cu")

# what must happen on the context's device: kernel launches, allocations, clears, and the functions that do them
NEEDS_DEVICE = re.compile(r"\blaunch\w+\s*[<(]|\bcheckLaunch\(|\.(?:reserve|resize|upload)\(|\bcudaMemsetAsync\(|\bcudaMalloc\w*\("
                          r"|\b(?:ensure\w+|buildBvh|uploadScene|publishScene|runPass|runParticles|castRays|materializePrims)\s*[<(]"
                          r"|\bcuda(?:Stream|Event)Create")


def entry_points():
    text = open(SOURCE).read()
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    out = {}
    for m in re.finditer(r"^int (owec_\w+)\([^)]*\)\s*\{", text, re.M):
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        out[m.group(1)] = text[m.end():k]
    return out


def test_entry_points_select_their_device():
    found = entry_points()
    assert len(found) > 25 and "owec_walk_resolve" in found
    late = []
    for name, body in found.items():
        need = NEEDS_DEVICE.search(body)
        device = body.find("cudaSetDevice(")
        if need and not 0 <= device < need.start():
            late.append(f"{name}: {need.group(0)}")
    assert not late, late
