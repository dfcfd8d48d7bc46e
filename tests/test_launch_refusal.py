"""A stencil launch that lacks an array its kernels read is refused on the host, before any
device call (no GPU needed): the passes of a handle, of a batch and of a residual-driven solve."""
import subprocess


MAIN = r"""
#include <cstdio>
#include <vector>
#include "fs_internal.cuh"
using namespace fs;
int main() {
    float* const some = reinterpret_cast<float*>(4096);  // never dereferenced
    int wrong = 0;
    auto expect = [&](cudaError_t e, const char* what) {
        if (e != cudaErrorInvalidValue) wrong += std::printf("%s: %s\n", what, cudaGetErrorName(e));
    };
    for (int kind : {PASS_DIFFUSE_FIRST, PASS_DIFFUSE, PASS_PRESSURE_FIRST, PASS_PRESSURE})
        for (int lacks = 0; lacks < 2; ++lacks)
            for (int rows : {64, 128})
                for (float* base : {some, some + 1}) {  // 16-byte rows or not
                    StencilField f{};
                    field_tiling(f, 130, 130, 160, rows, 2);
                    f.kind = kind;
                    f.sweeps = 2;
                    f.y = base;
                    const bool first = kind == PASS_DIFFUSE_FIRST || kind == PASS_PRESSURE_FIRST;
                    if (lacks != 0) f.x = base;
                    if (lacks != 1) (first ? f.x2 : f.cst) = base;
                    StencilLaunch L{};
                    L.nfields = 1;
                    L.f[0] = f;
                    expect(launch_stencil(L, rows, nullptr), "launch_stencil");
                    auto W = std::vector<WideLaunch>(1);
                    W[0] = {};
                    W[0].nfields = 1;
                    W[0].f[0] = f;
                    expect(prepare_stencil_wide(W[0]), "prepare_stencil_wide");
                }
    for (int lacks = 0; lacks < 5; ++lacks) {
        PressureSolve P{};
        field_tiling(P.mid, 130, 130, 160, 64, 9);
        P.mid.kind = PASS_PRESSURE;
        P.mid.sweeps = 8;
        P.first = P.mid;
        P.first.kind = PASS_PRESSURE_FIRST;
        P.max_passes = 1;
        if (lacks != 0) P.first.x = some;
        if (lacks != 1) P.first.x2 = some;
        if (lacks != 2) P.mid.cst = some;
        if (lacks != 3) P.p[0] = some;
        if (lacks != 4) P.p[1] = some;
        expect(launch_pressure_solve(P, 64, 1, nullptr), "launch_pressure_solve");
    }
    return wrong != 0;
}
"""


def test_a_launch_without_an_input_is_refused(fluid, tmp_path):
    from fluid2d_gb300 import build_lib as b

    src = tmp_path / "main.cu"
    src.write_text(MAIN)
    exe = tmp_path / "main"
    objects = [str(b.OBJ / (s.stem + ".o")) for s in b.sources()]
    r = subprocess.run([b.nvcc(), *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", f"-I{b.CSRC}", f"-I{b.INCLUDE}",
                        "-cudart", "static", str(src), *objects, "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
