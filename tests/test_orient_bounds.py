"""The source words an orientation tile reads and the kernel a surface takes, on
the CPU: the kernel's own
index arithmetic (csrc/orient_tile.h), built with the host compiler and walked
over every tile and row.  A tile that may read whole aligned words reads none
outside the caller's surface, at widths and heights of whole tiles and one or
two pixels more, on surfaces one and two pixels wide, and from every byte of a
word."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "jxr_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "orient_tile.h"
using namespace jxr;
// tile sides and the unit of aligned loads, as the kernels of each pixel size have them
int main(int argc, char **argv) {
    const uint32_t pb = (uint32_t)atoi(argv[1]), side = pb <= 4 ? 64 : 32;
    const uintptr_t step = pb % 2 == 0 ? 2 : 1;
    unsigned long outside = 0, words = 0, bytes = 0;
    const uint32_t extents[] = {1, 2, 3, 31, 33, 63, 64, 65, 66, 67, 127, 128, 129, 130, 193, 194};
    for (uint32_t w : extents)
        for (uint32_t h : extents)
            for (int o = 0; o < 8; o++)
                for (uintptr_t src = 4096; src < 4100; src += step) {
                    const uint64_t pitch = (uint64_t)w * pb, size = pitch * h;
                    const uint32_t ow = swaps_axes(o) ? h : w, oh = swaps_axes(o) ? w : h;
                    for (uint32_t dy = 0; dy < oh; dy += side)
                        for (uint32_t dx = 0; dx < ow; dx += side) {
                            const OrientTile t = orient_tile(o, w, h, side, dx, dy);
                            const uint64_t offset = t.sy0 * pitch + (uint64_t)t.sx0 * pb;
                            const uintptr_t first = src + offset;
                            if (t.sx0 + t.sw > w || t.sy0 + t.sh > h) { puts("rectangle"); return 1; }
                            const int n = t.sw * (int)pb;
                            if (!words_inside(src, size, offset, pitch, n, t.sh)) { bytes++; continue; }
                            words++;
                            for (int r = 0; r < t.sh; r++) {
                                const uintptr_t row = first + r * pitch;
                                const uintptr_t from = row & ~(uintptr_t)3, to = (row + n + 3) & ~(uintptr_t)3;
                                outside += from < src || to > src + size;
                            }
                        }
                }
    printf("%lu %lu %lu\n", outside, words, bytes);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("orient_bounds")
    (d / "bounds.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), str(d / "bounds.cpp"), "-o", str(d / "bounds")], check=True)
    return d / "bounds"


@pytest.mark.parametrize("pixel_bytes", [1, 2, 3, 6])
def test_word_reads_stay_inside_the_surface(program, pixel_bytes):
    out = subprocess.run([str(program), str(pixel_bytes)], check=True, capture_output=True, text=True).stdout
    outside, words, by_byte = map(int, out.split())
    assert outside == 0
    assert words > 0 and by_byte > 0


ROUTES = r"""
#include <cstdio>
#include <cstdlib>
#include "orient_tile.h"
int main(int argc, char **argv) {
    for (int i = 1; i + 3 < argc; i += 4)
        printf("%d\n", (int)jxr::takes_pixel_kernel(atoi(argv[i]), atoi(argv[i + 1]), atoi(argv[i + 2]), atoi(argv[i + 3])));
    return 0;
}
"""


def test_surfaces_of_each_kernel(tmp_path):
    """Pixels of 1 to 3 bytes from an extent on, every size from a narrower side
    on, at the alignment of their unit; other sizes never."""
    (tmp_path / "routes.cpp").write_text(ROUTES)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(tmp_path / "routes.cpp"), "-o", str(tmp_path / "routes")],
                   check=True)
    cases = []
    for n, extent, side in [(1, 1 << 20, 12), (2, 5 << 18, 16), (3, 3 << 17, 8), (4, 0, 12), (6, 0, 12), (8, 0, 8), (12, 0, 8),
                            (16, 0, 8)]:
        big = max(extent, 1 << 12)
        for w, h, taken in [(1 << 11, -(-big // (1 << 11)) + side, 1), (side, -(-big // side), 1), (-(-big // side), side, 1),
                            (side - 1, 2 * big, 0), (2 * big, side - 1, 0), (1, 2 * big, 0)]:
            cases.append((n, 0, w, h, taken))
        if extent:
            cases += [(n, 0, extent // 1024, 1023, 0), (n, 0, extent // 1024, 1024, 1)]
        if n % 2 == 0:
            cases += [(n, 1, 4096, 4096, 0), (n, 2, 4096, 4096, int(n % 4 != 0))]
    cases += [(n, 0, 4096, 4096, 0) for n in (5, 7, 10, 20, 48)]
    args = [str(v) for c in cases for v in c[:4]]
    out = subprocess.run([str(tmp_path / "routes"), *args], check=True, capture_output=True, text=True).stdout.split()
    assert [(c, int(o)) for c, o in zip(cases, out)] == [(c, c[4]) for c in cases]
