"""The colour-split layout's 32-bit byte offsets on grids up to the largest it
takes (2^31 cells), on the CPU: no signed overflow in forming them, and every
neighbour lands where 64-bit arithmetic puts it."""

import pathlib
import subprocess

CSRC = pathlib.Path(__file__).resolve().parent.parent / "stable-fluids_b200" / "csrc"

SOURCE = """
#include "sf_half_offsets.h"
#include <cstdio>
using sfb::Dims;
template <int B>
long check(Dims d, bool px, bool py, bool pz) {
    const long long hx = d.nx / 2, ny = d.ny, nz = d.nz;
    const long long ys[] = {0, 1, ny / 2, ny - 1}, zs[] = {0, 1, nz / 2, nz - 1}, ks[] = {0, 4, hx / 8 * 4, hx - 4};
    long wrong = 0;
    for (long long y : ys)
        for (long long z : zs)
            for (long long k0 : ks) {
                if (y < 0 || y >= ny || z < 0 || z >= nz || k0 < 0 || k0 + 4 > hx) continue;
                const auto o = sfb::half_offsets<B>(d, static_cast<int>(y), static_cast<int>(k0), px, py, pz);
                const long long at = B * (k0 + hx * (y + ny * z));
                const uint32_t i = static_cast<uint32_t>(at);
                const auto here = [&](uint32_t off, long long k, long long yy, long long zz) { wrong += static_cast<uint32_t>(i + off) != B * (k + hx * (yy + ny * zz)); };
                const auto near = [](long long c, long long n, bool p) { return c < 0 ? (p ? c + n : -1) : (c >= n ? (p ? c - n : -1) : c); };
                const long long yl = near(y - 1, ny, py), yh = near(y + 1, ny, py), zl = near(z - 1, nz, pz), zh = near(z + 1, nz, pz), kl = near(k0 - 1, hx, px), kh = near(k0 + 4, hx, px);
                here(o.y_lo, k0, yl < 0 ? y : yl, z);
                here(o.y_hi, k0, yh < 0 ? y : yh, z);
                here(z == 0 ? o.wrap : 0u - o.plane, k0, y, zl < 0 ? z : zl);
                here(z == nz - 1 ? 0u - o.wrap : o.plane, k0, y, zh < 0 ? z : zh);
                here(o.x_lo, kl < 0 ? k0 : kl, y, z);
                here(o.x_hi, kh < 0 ? k0 + 3 : kh, y, z);
            }
    return wrong;
}
int main() {
    const Dims grids[] = {{8, 2, 2, 0}, {16, 7, 5, 0}, {1024, 1024, 1024, 0}, {2040, 1024, 1026, 0}, {1280, 1290, 1300, 0}, {32768, 65528, 1, 0}, {65528, 2, 16384, 0}, {8, 2, 134217726, 0}, {8, 134217726, 2, 0}};
    long wrong = 0;
    for (const auto& d : grids)
        for (int p = 0; p < 8; ++p) wrong += check<4>(d, p & 1, p & 2, p & 4) + check<2>(d, p & 1, p & 2, p & 4);
    std::printf("%ld\\n", wrong);
    return 0;
}
"""


def test_offsets_up_to_the_largest_grid(tmp_path):
    (tmp_path / "offsets.cpp").write_text(SOURCE)
    exe = tmp_path / "offsets"
    subprocess.run(["g++", "-std=c++20", "-O1", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all", f"-I{CSRC}", str(tmp_path / "offsets.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["0"]
