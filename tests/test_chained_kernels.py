"""Kernels that start while the one before them still runs (those that call
chain_wait, csrc/common.cuh): the kernel before writes fields during their
lifetime, so they and the functions they share must not promise the compiler
that a field is constant or unaliased.  Read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stzpp_gb300", "csrc")
SETUP_ONLY = {"ainv", "nat_slot"}   # written by set-ups, never by a kernel of the cycle


def code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def functions(text):
    """(name, parameters, body) of the functions that have a body."""
    for m in re.finditer(r"(\w+)\(", text):
        i, depth = m.end(), 1
        while i < len(text) and depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, rest = text[m.end():i - 1], re.match(r"\s*\{", text[i:])
        if not rest or m.group(1) in ("if", "for", "while", "switch"):
            continue
        j, depth = i + rest.end(), 1
        while j < len(text) and depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), params, text[i + rest.end():j - 1]


def chained():
    found = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for name, params, body in functions(code(path)):
            if "chain_wait()" in body and name.endswith("_kernel"):
                found[name] = (os.path.basename(path), params, body)
    return found


def test_every_chained_launch_is_of_a_kernel_that_waits():
    launched = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = code(path)
        for m in re.finditer(r"launch_chained\((\w+)", text):
            name = m.group(1)
            if name == "kern":   # auto kern = name<...>, the last before the launch
                name = re.findall(r"auto kern = (\w+)", text[:m.start()])[-1]
            launched.add(name)
    assert launched and launched == set(chained())


@pytest.mark.parametrize("name", sorted(chained()))
def test_fields_are_not_promised_constant(name):
    path, params, _ = chained()[name]
    promised = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert promised <= SETUP_ONLY, (path, promised)


def test_functions_they_call():
    promising = {name for path in glob.glob(os.path.join(CSRC, "*.cuh")) for name, params, _ in functions(code(path))
                 if "__restrict__" in params}
    bodies = {name: body for name, (_, _, body) in chained().items()}
    for path in ("band.cu", "dense.cu", "plane.cu"):   # these hold nothing else
        for name, params, body in functions(code(os.path.join(CSRC, path))):
            assert "__restrict__" not in params, name
            bodies[name] = body
    for name, body in bodies.items():
        called = set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\(", body))
        assert not called & promising, (name, called & promising)
        # loads with a cache hint that nothing orders behind the waits
        assert not called & {"__ldcg", "__ldcs", "__ldca", "__ldlu", "__ldcv"}, name
