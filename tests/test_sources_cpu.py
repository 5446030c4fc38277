"""Rules that the CUDA sources have to keep and that no output shows."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bgk3d_hit_b200", "csrc")


def _functions():
    """name -> (signature, body) of every device function and kernel."""
    out = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in re.finditer(r"\b(__global__|__device__)\b[^;{}=]*?(\w+)\s*\((?=[^;]*?\)\s*\{)", text):
            b = text.find("{", m.end())
            depth, e = 0, b
            while True:
                depth += {"{": 1, "}": -1}.get(text[e], 0)
                if depth == 0:
                    break
                e += 1
            name = m.group(2)
            sig, body = out.get(name, ("", ""))
            out[name] = (sig + text[m.start():b], body + text[b:e])
    return out


def test_overlapped_kernels_read_with_ordinary_loads():
    """A kernel that starts beside the end of the one before it (step_begin) must not
    read by the read-only path, which wants data that nothing writes while the kernel
    is resident; nor may a function that it calls."""
    fn = _functions()
    kernels = [n for n, (_, b) in fn.items() if "step_begin();" in b]
    assert len(kernels) >= 14, kernels
    seen, todo = set(), list(kernels)
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        sig, body = fn[n]
        assert not re.search(r"\b_*ldg\w*\(|ld\.global\.nc|__restrict__", sig + body), n
        todo += [m for m in set(re.findall(r"\b(\w+)\s*(?:<[^;(]*>)?\(", body)) if m in fn]
    assert "aa_cell" in seen and "u16_at" in seen
