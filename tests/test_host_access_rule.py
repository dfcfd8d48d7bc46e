"""When kernels may address the caller's host grids (no GPU needed): only where the device reads
pageable memory through the host's own page tables, checked against a stand-in for the query."""
import os
import subprocess

import pytest

MAIN = r"""
#include "host_common.h"
namespace fs { int record_error(int code, const char*) { return code; } }
int main() { return fs::addresses_host(0) ? 10 : 20; }
"""
# the runtime's query, answered from the environment (attributes by their numbers)
FAKE = r"""
#include <cstdlib>
extern "C" int cudaDeviceGetAttribute(int* value, int attribute, int) {
    const char* name = attribute == 88 ? "PAGEABLE" : attribute == 100 ? "TABLES" : nullptr;
    const int v = name ? std::atoi(std::getenv(name)) : 0;
    if (v < 0) return 1;
    *value = v;
    return 0;
}
"""


@pytest.fixture(scope="module")
def rule(fluid, tmp_path_factory):
    from fluid2d_gb300 import build_lib as b

    d = tmp_path_factory.mktemp("rule")
    (d / "main.cu").write_text(MAIN)
    (d / "fake.cpp").write_text(FAKE)
    exe = d / "main"
    r = subprocess.run([b.nvcc(), *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", f"-I{b.CSRC}", f"-I{b.INCLUDE}",
                        "-cudart", "shared", str(d / "main.cu"), str(d / "fake.cpp"), "-o", str(exe), "-Xlinker", "-rpath", "-Xlinker",
                        str(b.pathlib.Path(b.nvcc()).resolve().parents[1] / "lib64")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return lambda pageable, tables: subprocess.run(
        [str(exe)], timeout=60, env={**os.environ, "PAGEABLE": str(pageable), "TABLES": str(tables)}).returncode == 10


def test_host_page_tables_are_required(rule):
    assert rule(1, 1)
    assert not rule(1, 0)  # software faults and migration
    assert not rule(0, 0) and not rule(0, 1)


def test_a_query_that_fails_means_no(rule):
    assert not rule(-1, 1) and not rule(1, -1)
