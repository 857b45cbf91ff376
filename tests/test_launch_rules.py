"""The rules that choose between kernels with the same results (sd3.c_b200/csrc/launch_rules.h): sizes that were timed on
both sides get the kernel that was faster.  148 SMs."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sd3.c_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text("""
#include <stdio.h>
#include "launch_rules.h"
int main() {
  char what; long a, b, c, d, e;
  while (scanf(" %c %ld %ld %ld %ld %ld", &what, &a, &b, &c, &d, &e) == 6)
    if (what == 'n') printf("%d\\n", static_cast<int>(sd3::ln_kernel(static_cast<int>(a), b, c != 0, 148)));
    else printf("%d\\n", sd3::pair_tile_width(a, b, static_cast<int>(c), d != 0, e != 0, 74));
}
""")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "rules.cpp"), "-o", str(d / "rules")],
                   check=True)

    def ask(queries):
        r = subprocess.run([str(d / "rules")], input="\n".join(queries), capture_output=True, text=True, check=True)
        return [int(v) for v in r.stdout.split()]
    return ask


WARP, CTA, ROWS = 0, 1, 2


def test_layernorm(rules):
    cases = [(64, 333, 0, CTA), (64, 1357, 0, WARP), (64, 35432, 0, WARP), (128, 589, 1, WARP), (128, 4429, 1, WARP),
             (256, 13287, 0, WARP), (260, 589, 1, ROWS), (512, 77, 0, CTA), (512, 3000, 0, WARP), (512, 3000, 1, WARP),
             (512, 13287, 0, WARP), (768, 589, 0, CTA), (768, 888, 0, WARP), (768, 35432, 1, WARP),
             (1024, 77, 1, ROWS), (1024, 3000, 0, CTA), (1024, 4429, 1, ROWS), (1024, 8858, 0, WARP), (1024, 17000, 0, WARP),
             (1280, 8858, 0, WARP), (1280, 9500, 0, ROWS), (1280, 35432, 1, ROWS),
             (1536, 77, 0, CTA), (1536, 3000, 0, CTA), (1536, 4429, 0, WARP), (1536, 8200, 0, ROWS), (1536, 35432, 0, ROWS),
             (1536, 589, 1, ROWS), (1536, 35432, 1, ROWS), (1540, 77, 0, WARP), (2432, 4429, 1, WARP)]
    assert rules(["n %d %d %d 0 0" % c[:3] for c in cases]) == [c[3] for c in cases]


def test_tile_width(rules):
    def q(rows, N, K, gate, after=0, fp8=0):
        tiles = (rows + 255) // 256 * (N // 256)
        return "w %d %d %d %d %d" % (tiles + after, after, K, fp8, gate)
    cases = [(q(589, 4608, 1536, 0), 128), (q(1357, 4608, 1536, 0), 128), (q(2714, 4608, 1536, 0), 256),
             (q(4429, 4608, 1536, 0), 256), (q(1024, 6144, 1536, 0), 128), (q(1357, 6144, 1536, 0), 256),
             (q(256, 1536, 6144, 1), 64), (q(700, 1536, 6144, 1), 64), (q(2714, 1536, 6144, 1), 256),
             (q(4429, 1536, 6144, 1), 128), (q(5428, 1536, 6144, 1), 256), (q(4429, 1536, 1536, 1), 128),
             (q(1332, 1536, 4096, 0), 128),
             # few K blocks, several waves
             (q(8192, 1024, 1024, 1), 256), (q(16384, 1024, 1024, 0), 256), (q(16384, 512, 512, 1), 256),
             (q(8192, 1536, 512, 0), 256), (q(2714, 1024, 1024, 0), 128), (q(4096, 1536, 512, 1), 128),
             # FP8, 576 + 333 tokens: QKV (three problems) and MLP1
             (q(2 * 768 + 512, 4608, 1536, 0, fp8=1), 128), (q(768 + 512, 6144, 1536, 0, fp8=1), 128),
             # a dual block's out-projections: 256 + 333, 1024 + 333 and 4096 + 333 rows
             (q(256 + 512, 1536, 1536, 1, after=6), 64), (q(1024 + 512, 1536, 1536, 1, after=24), 128),
             (q(4096 + 512, 1536, 1536, 1, after=96), 128)]
    assert rules([c[0] for c in cases]) == [c[1] for c in cases]
