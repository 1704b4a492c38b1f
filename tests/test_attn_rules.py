"""Which attention kernel a call's sizes ask for (csrc/attn_rules.h), held against measured times of both kernels on a B200."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "umbrella_b200", "csrc")
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")

    def go(call, values):
        src = "#include <cstdio>\n#include \"attn_rules.h\"\nint main() {\n" + "".join(f'printf("%d\\n", (int)umb::{call}({", ".join(map(str, v))}, 148));\n' for v in values) + "}\n"
        (d / "a.cpp").write_text(src)
        subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "a.cpp"), "-o", str(d / "a")], check=True)
        return [bool(int(x)) for x in subprocess.run([str(d / "a")], check=True, capture_output=True, text=True).stdout.split()]
    return go


# (blocks, keys): us with four warps, with six; 8 heads or fewer to a block, of 128, 96 and 64
DECODE = {(74, 1201): (19.6, 19.6), (148, 301): (15.9, 12.1), (152, 101): (9.6, 9.9), (152, 301): (18.2, 15.7), (200, 201): (14.1, 15.0), (256, 101): (9.9, 10.3),
          (256, 201): (14.2, 15.4), (256, 301): (18.8, 16.1), (256, 1201): (47.6, 41.4), (296, 2001): (72.0, 63.2), (304, 31): (9.7, 16.2), (304, 501): (26.2, 34.0),
          (400, 201): (16.2, 27.8), (400, 1201): (56.8, 77.6), (400, 2001): (86.0, 106.0), (512, 301): (38.0, 30.0), (512, 2001): (151.0, 119.0), (592, 301): (39.0, 31.0),
          (592, 2001): (152.0, 120.0), (800, 201): (29.8, 41.0), (800, 1201): (109.0, 116.0), (1024, 31): (25.0, 32.4), (1024, 201): (45.0, 57.0), (1024, 501): (72.0, 77.0),
          (1024, 2001): (231.0, 217.0), (2048, 201): (76.0, 100.0), (2048, 501): (123.0, 135.0), (2048, 2001): (392.0, 402.0)}


def test_warps_of_a_decode_block(ask):
    """Never more than 3 % behind the better one where six warps are taken, nor 7 % where four are."""
    for (at, (four, six)), took_six in zip(DECODE.items(), ask("six_warps_pay", DECODE)):
        assert (six <= 1.03 * four) if took_six else (four <= 1.07 * six), (at, four, six)


# (mask mode, rows, keys, heads, key/value heads, head size): us in slabs of 16 rows, in tiles of 64
ROWS = {(2, 256, 256, 32, 8, 128): (18.4, 15.3), (2, 256, 7256, 32, 8, 128): (204.8, 172.6), (2, 128, 628, 64, 8, 128): (34.8, 29.1), (2, 300, 300, 32, 8, 128): (27.9, 17.2),
        (2, 300, 1800, 32, 8, 128): (76.2, 82.9), (2, 300, 7300, 32, 8, 128): (253.0, 320.0), (2, 296, 7296, 32, 8, 128): (211.0, 320.0), (2, 512, 512, 32, 8, 128): (49.0, 28.0),
        (2, 512, 7512, 32, 8, 128): (367.0, 331.0), (2, 520, 7520, 32, 8, 128): (410.0, 332.0), (2, 600, 600, 32, 8, 128): (60.0, 33.0), (2, 600, 3100, 32, 8, 128): (200.0, 208.0),
        (2, 600, 7600, 32, 8, 128): (459.0, 546.0), (2, 512, 512, 64, 8, 128): (91.0, 43.0), (2, 192, 7192, 64, 8, 128): (302.0, 317.0), (2, 1000, 8000, 32, 32, 128): (799.0, 688.0),
        (0, 512, 1012, 64, 8, 128): (162.0, 124.0), (0, 256, 1256, 64, 8, 128): (92.0, 66.0), (0, 300, 7300, 32, 8, 128): (261.0, 331.0), (0, 800, 1300, 32, 8, 128): (163.0, 170.0),
        (0, 800, 1300, 24, 8, 128): (130.0, 169.0), (0, 400, 900, 32, 8, 128): (68.0, 57.0), (1, 300, 2300, 32, 8, 128): (235.0, 387.0), (1, 300, 800, 64, 8, 128): (199.0, 248.0),
        (2, 256, 256, 32, 8, 64): (9.1, 10.9), (2, 300, 300, 32, 8, 64): (17.0, 12.0), (2, 512, 512, 32, 8, 64): (30.0, 22.0), (2, 512, 1512, 32, 8, 64): (57.0, 61.0),
        (2, 384, 7384, 32, 8, 64): (175.0, 265.0), (0, 384, 4384, 32, 8, 64): (117.0, 169.0), (2, 768, 7768, 16, 16, 64): (180.0, 278.0), (2, 600, 600, 16, 16, 64): (21.0, 23.0)}


def test_rows_of_an_attention_block(ask):
    """Never more than 2 % behind the better one where tiles are taken, nor 10 % where slabs are."""
    for (at, (slabs, tiles)), took in zip(ROWS.items(), ask("row_tiles_pay", ROWS)):
        assert (tiles <= 1.02 * slabs) if took else (slabs <= 1.1 * tiles), (at, slabs, tiles)
