"""Shared arrays that kernels read or write by vectors, or fill by 16-byte
asynchronous copies, state the alignment they need: without __align__ an array of
float or double is only sure to have its element's (read from the sources)."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "tabi-pb_b200", "csrc")
WIDTH = {"float2": 8, "float4": 16, "double2": 16, "double4": 16, "int2": 8, "int4": 16}
ELEM = {"float": 4, "double": 8, "int": 4}


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for part in re.split(r"(?m)^(?=.*__global__)", open(path).read()):
            yield os.path.basename(path), part


def _shared(part):
    """(name, alignment, extern) of the shared arrays of scalars."""
    pat = r"(extern )?__shared__ (?:__align__\((\d+)\) )?(float|double|int) ([^;]+);"
    for ext, align, typ, names in re.findall(pat, part):
        for name in re.findall(r"(\w+)\s*(?=\[)", re.sub(r"\[[^\]]*\]", "[]", names)):
            yield name, int(align) if align else ELEM[typ], bool(ext)


def test_vector_accesses_to_shared_arrays():
    seen = 0
    for path, part in _kernels():
        for name, align, ext in _shared(part):
            for vec in re.findall(rf"reinterpret_cast<(?:const )?(\w+)\*>\(&?{name}\b", part):
                seen += 1
                assert align >= WIDTH[vec], (path, name, vec)
            if ext and "cp_async16" in part:
                assert align >= 16, (path, name)
    assert seen >= 5
