"""The host side of the C entry points on a stand-in for the CUDA runtime (tests/support/host_calls.cpp): what
depends on several devices, on allocations that fail or on solves that give up, without a GPU."""

import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "opensurgsim_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    """gbfem_host.cpp and gbfem_plan.cpp linked with the stand-in; kernels and CUDA calls that it leaves out do
    nothing and return 0."""
    from opensurgsim_gb300 import build

    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    if not all(map(shutil.which, ("g++", "gcc", "nm"))) or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("the compilers or the CUDA headers are missing")
    out = str(tmp_path_factory.mktemp("host_calls"))
    sources = [os.path.join(CSRC, "gbfem_host.cpp"), os.path.join(CSRC, "gbfem_plan.cpp"),
               os.path.join(ROOT, "tests", "support", "host_calls.cpp")]
    objects = [os.path.join(out, os.path.basename(s) + ".o") for s in sources]
    limit = os.path.join(out, "limit.h")  # the range of 32-bit indices as a variable
    with open(limit, "w") as f:
        f.write("#include <cstdint>\n#undef INT32_MAX\nextern long long fake_int32_max;\n#define INT32_MAX fake_int32_max\n")
    jobs = [subprocess.Popen(["g++", "-c", "-include", limit, "-w", "-g", "-O0", "-std=c++17", "-fsanitize=address", "-I" + CSRC, "-I" + cuda, s,
                              "-o", o]) for s, o in zip(sources, objects)]
    assert [j.wait() for j in jobs] == [0, 0, 0]
    symbols = {kind: set() for kind in "UT"}
    for line in subprocess.run(["nm"] + objects, capture_output=True, text=True, check=True).stdout.splitlines():
        m = re.match(r"\S*\s+([A-Za-z])\s+(\S+)$", line)
        if m:
            symbols["U" if m[1] == "U" else "T"].add(m[2])
    missing = sorted(s for s in symbols["U"] - symbols["T"] if re.match(r"_ZN5gbfem|cuda[A-Z]", s))
    stubs = os.path.join(out, "stubs.c")
    with open(stubs, "w") as f:
        f.writelines(f"long {s}(void) {{ return 0; }}\n" for s in missing)
    exe = os.path.join(out, "host_calls")
    subprocess.run(["gcc", "-c", "-w", stubs, "-o", stubs + ".o"], check=True)
    subprocess.run(["g++", "-fsanitize=address", "-o", exe, stubs + ".o"] + objects, check=True)
    return exe


@pytest.mark.parametrize("case", ["two_devices", "failed_allocations", "failed_host_memory", "errors_reported_once",
                                  "positions_without_an_order", "patience", "index_range"])
def test_host_calls(program, case):
    out = subprocess.run([program, case], capture_output=True, text=True, env={**os.environ, "ASAN_OPTIONS": "detect_leaks=0"})
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_the_benchmark_gives_no_hbm_fraction_of_a_resident_solve():
    import bench

    far = bench.solve_roofline(False, 123, 3000.0, 6000.0)
    assert "k_pcg_persistent" in far["kernel"] and far["bound"] == "hbm" and far["frac"] == 0.5 and far["traffic"] == 123
    near = bench.solve_roofline(True, 123, 9000.0, 6000.0)
    assert "k_res" in near["kernel"] and near["frac"] is None and near["traffic"] is None and near["achieved"] == 9000.0
