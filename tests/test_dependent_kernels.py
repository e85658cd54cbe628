"""Kernels that are launched while the kernel before them still runs
(launch_dependent) must not read what that kernel writes through the read-only
path: it is valid only for memory that nobody writes from the launch on, and
the compiler may move such loads to before the wait.  Which path a load takes
cannot be seen from results, so this reads the sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eshwar_dipan_b200", "csrc")
# written by the host only, before any step
CONSTANT = {"sims", "consts", "tsim", "tmaps"}


def _sources():
    text = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))):
        if "adjoint" not in f and "dual" not in f:   # ordinary launches
            with open(f) as h:
                text[os.path.basename(f)] = re.sub(r"/\*.*?\*/|//[^\n]*", "", h.read(), flags=re.S)
    return text


def _functions(src):
    """(name, parameters, body) of every device function and kernel."""
    for m in re.finditer(r"__(?:global|device)__\s[^;{}]*?\b(\w+)\(", src):
        if m.group(1) in ("__launch_bounds__", "__align__"):
            continue
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(src[i], 0)
            i += 1
        params, rest = src[m.end():i - 1], src[i:].lstrip()
        if m.group(1) == "__launch_bounds__" or not rest.startswith("{"):
            continue
        j = i + len(src[i:]) - len(rest) + 1
        k, depth = j, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        yield m.group(1), params, src[j:k]


def _all():
    out = {}
    for src in _sources().values():
        flat = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", src)
        for name, params, body in _functions(flat):
            out.setdefault(name, []).append((params, body))
    return out


def _dependent(funcs):
    """the kernels launched by launch_dependent and every device function they reach"""
    kernels = {n for n, defs in funcs.items() if any("pdl_begin()" in b or "box_begin<" in b for _, b in defs)}
    seen, todo = set(), set(kernels)
    while todo:
        n = todo.pop()
        seen.add(n)
        for _, body in funcs[n]:
            todo |= {w for w in re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\(", body) if w in funcs} - seen
    return kernels, seen


def test_every_dependent_launch_waits():
    src = _sources()["gp_batch_impl.cuh"]
    launched = set(re.findall(r"launch_dependent\([\w.]+, (k\w+)<", src)) | set(re.findall(r"\bf\((k\w+)<", src))
    kernels, _ = _dependent(_all())
    assert {"kf_classify", "kf_bulk", "kf_general", "kf_step", "ks_tiles"} == launched == kernels


def test_no_read_only_pointers_to_stepped_memory():
    funcs = _all()
    _, reached = _dependent(funcs)
    assert {"general_tiles", "bulk_tiles", "bulk_phase", "smooth_cell", "tile32", "item_current"} <= reached
    bad = []
    for n in sorted(reached):
        for params, _ in funcs[n]:
            for p in re.findall(r"const\s+[\w:]+(?:<[^<>]*>)?\s*\*\s*__restrict__\s+(\w+)", params):
                if p not in CONSTANT and not (n == "bulk_cell_full_f64" and p in ("st", "Dp")):   # shared memory, constants
                    bad.append("%s: %s" % (n, p))
    assert not bad, bad


def test_no_read_only_loads_of_stepped_memory():
    funcs = _all()
    _, reached = _dependent(funcs)
    bad = []
    for n in sorted(reached):
        for _, body in funcs[n]:
            for arg in re.findall(r"__ldg\(([^()]*)", body):
                # the copy of a simulation's constants; the ordinary sweep's own path
                ok = re.match(r"(tsim|consts)\b", arg) or (n == "general_tiles" and arg == "src + w") or n == "ld_sweep"
                if not ok:
                    bad.append("%s: __ldg(%s)" % (n, arg))
    assert not bad, bad
