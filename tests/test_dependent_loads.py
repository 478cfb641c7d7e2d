"""Kernels that wait for the launch before them (programmatic dependent launch) start while that launch still runs: what it may be
writing is read with ordinary loads after the wait.  The read-only path (__ldg, ld.global.nc) is for memory that nothing writes
during the kernel's life, and the compiler may move such a load above the wait.  Checked in the source: no run shows it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paralleltnnlayers_b200", "csrc")
# The caller's factors, which no launch of the same call writes; the call's first launch is a plain one, so that every kernel before
# the call has completed.
FACTORS = {("cp4_grad_band.cu", "KH"), ("cp4_grad_band.cu", "KW"), ("cp4_grad_band.cu", "src"), ("cp_planes.cu", "src")}


def _functions(text):
    """name -> (parameters, body) of every device function and kernel that is defined in a source"""
    text = re.sub(r"//[^\n]*", "", text)
    found = {}
    for m in re.finditer(r"__global__|__device__", text):
        head = re.compile(r"[^{};]*\{").match(text, m.end())
        if not head or ")" not in head.group(0):
            continue
        sig = head.group(0)
        close = sig.rindex(")")
        depth, at = 1, close   # back to the parenthesis that opens the parameters
        while depth:
            at -= 1
            depth += {")": 1, "(": -1}.get(sig[at], 0)
        name = re.search(r"(\w+)\s*$", sig[:at])
        depth, i = 1, head.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        if name:
            found[name.group(1)] = (sig[at:close], text[head.end():i])
    return found


def _reach(functions, name):
    seen, todo = set(), [name]
    while todo:
        n = todo.pop()
        if n not in seen:
            seen.add(n)
            todo += [w for w in set(re.findall(r"\b(\w+)\s*[<(]", functions[n][1])) if w in functions]
    return seen


def test_waiting_kernels_read_with_ordinary_loads():
    kernels, bad = 0, []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        functions, file = _functions(open(path).read()), os.path.basename(path)
        for name, (params, body) in functions.items():
            if "grid_dependency_wait()" not in body:
                continue
            kernels += 1
            for p in params.split(","):   # const and restrict, read in C (not as the address of a copy): the read-only path again
                word = p.split()[-1]
                read = re.search(r"\b%s\s*\[|\*\s*\(?%s\b|__ldg\(%s\b" % (word, word, word), body)
                if re.match(r"[(\s]*const\b.*__restrict__", p, re.S) and read and (file, word) not in FACTORS:
                    bad.append((file, name, p.strip()))
            for f in _reach(functions, name):
                for arg in re.findall(r"__ldg\(([^;]*)", functions[f][1]):
                    first = re.sub(r"reinterpret_cast<[^>]*>\(", "", arg)
                    if (file, re.match(r"[\w.]*", first).group(0)) not in FACTORS:
                        bad.append((file, name, f, arg[:40]))
    assert kernels >= 15
    assert not bad, bad
