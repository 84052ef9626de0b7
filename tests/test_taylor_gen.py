"""The generated far-field header: in line with its generator, and refused for
other than FP32, whose moments it reads."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "tabi-pb_b200", "csrc")


def test_header_is_the_generators(tmp_path):
    shutil.copy(os.path.join(CSRC, "gen_taylor.py"), tmp_path)
    subprocess.run([sys.executable, str(tmp_path / "gen_taylor.py"), "8"], check=True)
    assert (tmp_path / "taylor_gen.cuh").read_bytes() == \
        open(os.path.join(CSRC, "taylor_gen.cuh"), "rb").read()


@pytest.mark.parametrize("typ", ["float", "double"])
def test_header_is_single_precision(tmp_path, typ):
    src = tmp_path / "use.cu"
    src.write_text(f"""#include "taylor_gen.cuh"
__global__ void use({typ}* v, const float4* m) {{
  far_eval<1, {typ}>(v[0], v[1], v[2], v[3], m, v[4], v[5], v[6], v[7], v[8], v[9], v[10]);
}}
""")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    r = subprocess.run([nvcc, "-arch=sm_100a", "-std=c++17", "-I", CSRC, "-c", str(src), "-o",
                        str(tmp_path / "use.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == (typ == "float"), r.stderr
