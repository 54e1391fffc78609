"""Kernels whose launches take more shared memory than the default: their limit
is a property of the function on a device, shared by every thread of the
process.  Read from the sources: it is set in one place (SmemLimit of
csrc/launch.h), which marks it as set only after setting it and is given sizes
that no launch exceeds, never one launch's own."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stzpp_gb300", "csrc")


def code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def sources():
    return sorted(p for e in ("*.cu", "*.cuh", "*.h") for p in glob.glob(os.path.join(CSRC, e)))


def test_one_place_sets_limits():
    where = [os.path.basename(p) for p in sources() if "cudaFuncAttributeMaxDynamicSharedMemorySize" in code(p)]
    assert where == ["launch.h"]
    text = code(os.path.join(CSRC, "launch.h"))
    body = text[text.index("void allow("):]
    assert body.index("cudaFuncSetAttribute") < body.index("fetch_or")   # set, then marked as set


def test_limits_do_not_depend_on_a_launch():
    """The sizes given are constants of the build: of templates, or of the largest bottom."""
    seen = 0
    for p in sources():
        text = code(p)
        for m in re.finditer(r"\blimit\.allow\(|_limit\.allow\(", text):
            i, depth = m.end(), 1
            while depth and not (depth == 1 and text[i] == ","):
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            size = text[m.end():i].strip()
            if size == "smem":   # const int smem = ..., the last before it
                size = re.findall(r"const int smem = ([^;]*);", text[:m.start()])[-1]
            words = set(re.findall(r"[A-Za-z_]\w*", size))
            allowed = {"int", "sizeof", "double", "double2", "float", "T", "M2", "std", "max", "fourier_smem"}
            assert all(w in allowed or re.match(r"k[A-Z]\w*$|TileBuf$", w) for w in words), (p, size)
            seen += 1
    assert seen >= 9
