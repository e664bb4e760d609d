"""The numbering of neighbour cells on the host: every pair of neighbouring
cells of grids from one cell per direction up, thin ones in each direction, as
the kernels of the assembly number them (device code compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <cstdio>
#include "k_ppe.cuh"
template <int D>
static int check()
{
    int bad = 0, pairs = 0;
    for (int nx = 1; nx <= 5; nx++)
        for (int ny = 1; ny <= 5; ny++)
            for (int nz = 1; nz <= (D == 3 ? 4 : 1); nz++) {
                mps::Grid<D> g{};
                g.dims[0] = nx;
                g.dims[1] = ny;
                if (D == 3) g.dims[D - 1] = nz;
                for (int a = 0; a < nx * ny * nz; a++)
                    for (int b = 0; b < nx * ny * nz; b++) {
                        int x = b % nx - a % nx, y = b / nx % ny - a / nx % ny, z = b / (nx * ny) - a / (nx * ny);
                        if (x * x > 1 || y * y > 1 || z * z > 1) continue;
                        int want = x + 1 + 3 * (y + 1) + (D == 3 ? 9 * (z + 1) : 0);
                        bad += mps::neighbour_cell<D>(g, b, a) != want;
                        pairs++;
                    }
            }
    std::printf("%d-D: %d of %d pairs wrong\n", D, bad, pairs);
    return bad;
}
int main() { return check<2>() + check<3>() ? 1 : 0; }
'''


def test_every_neighbour_has_its_number(tmp_path):
    nvcc = os.environ.get("NVCC", "nvcc")
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "numbers.cu"
    src.write_text(SOURCE)
    exe = str(tmp_path / "numbers")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
                        "-I" + os.path.join(ROOT, "mps_b200", "csrc"), "-o", exe, str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
