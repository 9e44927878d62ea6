"""Kernels launched as programmatic dependent launches read what the kernel before
them wrote.  They wait for it before their first access to global memory, and
neither they nor what they call promise the compiler that memory is read-only
(__restrict__, __ldg): such a load could move before the wait."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "procedural-universe_gb300", "csrc")


def functions():
    """name -> [(signature, body)] of the device code's functions, comments left out."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"(?:__global__|__device__)[^;{}()]*(?:__launch_bounds__\([^()]*\)[^;{}()]*)?\b(\w+)\s*\(", text):
            at, depth = m.end(), 1
            while depth:   # the parameters
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            brace = re.match(r"\s*(?:const\s*)?\{", text[at:])
            if not brace:
                continue
            end, depth = at + brace.end(), 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out.setdefault(m.group(1), []).append((text[m.start():at], text[at:end]))
    return out


def launched_after():
    names = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"launch_after\(([^;]*?);", text, flags=re.S):
            names |= set(re.findall(r"\bk_\w+", m.group(1).split(", ")[0] + " " + m.group(1)[:200]))
    return names


def test_dependent_kernels_wait_first_and_promise_nothing():
    fns, kernels = functions(), launched_after()
    assert {"k_sort_pass", "k_link", "k_place", "k_mass", "k_kick_drift", "k_direct_rows", "k_direct_rows_update",
            "k_writeback_records"} <= kernels
    for kernel in sorted(kernels):
        assert all("wait_for_previous();" in body for _, body in fns[kernel]), kernel
        seen, todo = set(), [kernel]
        while todo:
            name = todo.pop()
            if name in seen:
                continue
            seen.add(name)
            for signature, body in fns[name]:
                assert "__restrict__" not in signature + body, (kernel, name)
                assert "__ldg" not in body, (kernel, name)
                todo += [w for w in set(re.findall(r"\b([a-z]\w*)\s*(?:<[^;(){}]*>)?\s*\(", body)) if w in fns]
