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
  char what; long a, b, c;
  while (scanf(" %c %ld %ld %ld", &what, &a, &b, &c) == 4)
    if (what == 'n') printf("%d\\n", static_cast<int>(sd3::ln_kernel(static_cast<int>(a), b, c != 0, 148)));
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
    assert rules(["n %d %d %d" % c[:3] for c in cases]) == [c[3] for c in cases]
