"""Which form of the 32-bit product a size takes: host logic alone, built without a GPU.  The sizes are ones at which both forms
were timed and lie further apart than the runs of one."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neurogrid_b200", "csrc")


def _ask(tmp_path, call, sizes):
    src, exe = tmp_path / "form.cpp", tmp_path / "form"
    src.write_text('#include "gemm_f32_form.h"\n#include <cstdio>\nint main() { int m, n, k; while (scanf("%d %d %d", &m, &n, &k) == 3) '
                   'printf("%d\\n", (int)' + call + '); return 0; }\n')
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], input="\n".join("%d %d %d" % s for s in sizes), check=True, capture_output=True, text=True).stdout
    return [int(v) for v in out.split()]


@pytest.mark.parametrize("cluster,sizes", [
    (False, [(1, 1024, 2048), (1, 3072, 2048), (1, 1024, 3072), (1, 2048, 3072), (1, 2048, 8192), (1, 16384, 2048), (2, 1024, 1536), (2, 2048, 2048), (2, 6144, 2048), (2, 9216, 1536),
             (3, 1536, 1536), (4, 2048, 2048), (8, 1024, 1536), (8, 1024, 2048), (16, 512, 1536), (8, 1024, 1024), (8, 1024, 9216)]),
    (True, [(1, 1024, 4608), (1, 1024, 8192), (1, 3072, 3072), (1, 4096, 8192), (2, 512, 1536), (2, 4800, 2048), (2, 16384, 2048), (2, 2048, 4608), (4, 3072, 2048),
            (4, 1536, 4608), (8, 256, 2048), (24, 256, 2048), (8, 1536, 1536), (8, 3072, 2048), (9, 1024, 2048), (32, 3072, 2048), (32, 65536, 2048)])])
def test_few_rows_take_the_faster_form(tmp_path, cluster, sizes):
    assert dict(zip(sizes, _ask(tmp_path, "gf_rows_cluster(m, n, k)", sizes))) == {s: int(cluster) for s in sizes}


# (rows, columns, K): the tile (0: 64 x 64, 1: 32 x 64, 2: 32 x 32) and whether its groups are a cluster
TILES = {
    (33, 1024, 1024): (2, 0), (64, 1024, 1024): (2, 0), (96, 1536, 1024): (1, 0), (192, 1024, 1024): (1, 0), (1024, 1024, 1024): (0, 0),
    (192, 9216, 1024): (0, 0), (640, 1536, 1536): (0, 0), (96, 9216, 1536): (1, 0), (192, 9216, 1536): (0, 0), (2048, 3072, 1536): (0, 0),
    (256, 3072, 1536): (1, 0), (64, 3072, 1536): (1, 1), (1024, 1024, 1280): (0, 0), (128, 1024, 4608): (1, 1), (256, 512, 1024): (1, 0), (96, 3072, 1536): (1, 1), (192, 1024, 4608): (1, 1),
    (2048, 1024, 4608): (0, 0), (384, 2048, 2048): (0, 1), (1024, 3072, 2048): (0, 1), (2048, 2048, 2048): (0, 0), (640, 2048, 8192): (0, 1),
    (2048, 2048, 8192): (0, 0), (640, 2048, 3072): (0, 1), (256, 4096, 3072): (0, 0), (33, 2048, 9216): (2, 0), (96, 2048, 9216): (1, 0),
}


def test_tiles_take_the_faster_form(tmp_path):
    got = _ask(tmp_path, "(2 * gf_tile_size(m, n, k) + gf_tile_cluster(m, n, k))", list(TILES))
    assert {s: (v // 2, v % 2) for s, v in zip(TILES, got)} == TILES
