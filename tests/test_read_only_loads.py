"""Kernels that may start under the kernel before them (griddepcontrol.wait) read what that
kernel writes with plain loads.  __ldg and const __restrict__ promise data that are constant for
the reading kernel's whole life, which such a launch breaks, and a compiler may place the load
ahead of the wait.  Tables that no kernel writes while it runs may keep them."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turbchannel_b200", "csrc")
# twiddle factors; the z-solve's factors; the closure's parameters of a run (copied from the host)
TABLES = {"tw", "twx", "twy", "fac"}
PARAMETERS = {("k_turb_mlp", "P")}
SAMPLES = {("k_mlp_grad", "X"), ("k_mlp_grad", "Y")}  # copied from the host before training


def _functions(text):
    """(name, parameters, body) of every function defined at namespace level."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*(?:\([^()]*\))?[^()]*\))*\)", "", text)
    for m in re.finditer(r"^(?:template[^\n]*\n)?[^\n#]*?\b(\w+)\(", text, re.M):
        i, depth = m.end(), 1
        while depth and i < len(text):
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        brace = re.match(r"\s*\{", text[i:])
        if not brace:
            continue
        j, depth = i + brace.end(), 1
        while depth and j < len(text):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), text[m.end():i - 1], text[i:j]


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield os.path.basename(path), list(_functions(f.read()))


def test_kernels_behind_a_wait_read_plainly():
    found = 0
    for name, functions in _sources():
        for fn, params, body in functions:
            if fn == "pdl_wait" or "pdl_wait()" not in body:
                continue
            found += 1
            for p in re.findall(r"const\s+[\w<>: ]+\*\s*__restrict__\s+(\w+)", params):
                assert p in TABLES or (fn, p) in PARAMETERS | SAMPLES, f"{name}: {fn}({p})"
            for p in re.findall(r"const\s+[\w<>: ]+\*\s*__restrict__\s+(\w+)", body):
                assert p in TABLES, f"{name}: {fn}, local {p}"
            for p in re.findall(r"ldg_c\(\s*(\w+)", body):
                assert p in TABLES, f"{name}: {fn}, ldg_c({p})"
    assert found >= 15  # the functions are found at all


def test_ldg_is_for_tables():
    for name, functions in _sources():
        for fn, _, body in functions:
            if re.search(r"\b__ldg\(", body):
                # ldg_c: twiddle factors; k_flux_mlp: always an ordinary launch
                assert fn in ("ldg_c", "k_flux_mlp"), f"{name}: {fn}"
