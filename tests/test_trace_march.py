"""The march length of the tiled trace (trace_march, csrc/step_impl.cuh): the function is taken from the
header, compiled for the host and asked for grids of every shape.  The planes of a march are those of the grid
at most, and the marches of a column stay within the 65535 blocks a launch may have along z; where they would
not, a column of a million planes and a few cells across would be refused that one of a thousand is not."""
import pathlib
import re
import subprocess

CSRC = pathlib.Path(__file__).resolve().parents[1] / "dumses_hybrid_b200" / "csrc"

MAIN = """
#include <cstdio>
%s
int main() {
    int tiles, planes, slots;
    while (std::scanf("%%d %%d %%d", &tiles, &planes, &slots) == 3) std::printf("%%d\\n", trace_march(tiles, planes, slots));
}
"""


def test_march_fits_the_grid_and_the_launch(tmp_path):
    text = (CSRC / "step_impl.cuh").read_text()
    fn = re.search(r"constexpr double kTraceFill.*?^}\n", text, re.S | re.M).group(0)
    src, exe = tmp_path / "march.cpp", tmp_path / "march"
    src.write_text(MAIN % fn)
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", str(src), "-o", str(exe)], check=True)
    # planes: small ones, those of ordinary grids, columns up to the index limit of 2^31 ghosted cells (7 x 7 across)
    planes = list(range(1, 70)) + [130, 258, 514, 1026, 65535, 65536, 131072] + list(range(900000, 1100000, 101)) + \
        [2000000, 16 * 65535, 16 * 65535 + 1, 43000000]
    asked = [(t, p, s) for s in (592, 740) for t in (1, 2, 3, 5, 64, 4096, 70000) for p in planes]
    out = subprocess.run([str(exe)], input="".join("%d %d %d\n" % a for a in asked), capture_output=True, text=True, check=True)
    marches = list(map(int, out.stdout.split()))
    assert len(marches) == len(asked)
    for (tiles, n, slots), kz in zip(asked, marches):
        assert 1 <= kz <= n, (tiles, n, slots, kz)
        assert -(-n // kz) <= 65535, (tiles, n, slots, kz)
        assert kz <= 16 or n > 16 * 65535, (tiles, n, slots, kz)
