"""Which tiles of a grouped GEMM launch a CTA pair runs (sd3.c_b200/csrc/pair_tiles.h), walked on the host: where two
problems add to the same rows, one pair runs both tiles, so pairs never wait for each other."""
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sd3.c_b200", "csrc")


def test_tile_walk(tmp_path):
    exe = str(tmp_path / "model")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "pair_tiles_model.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_all_roles_of_the_kernel_take_this_walk():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gemm2_tcgen05.cu")).read())
    loops = re.findall(r"for \(int tile = pair;[^{]*\{", src)
    assert len(loops) == 3 and all("tile = tiles.next(tile, num_pairs)" in s for s in loops)


def test_no_kernel_waits_on_a_word_in_global_memory():
    """CTAs of a launch outside one cluster are not started together: a wait for another one may have no end."""
    for f in sorted(os.listdir(CSRC)):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        assert not re.search(r"ld\.(acquire|relaxed|volatile)[a-z0-9_.:]*\.(gpu|sys|global)", src), f
