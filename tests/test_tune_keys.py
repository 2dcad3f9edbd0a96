"""Which launches share a tuned shape, and which shape launches that share one take (host code,
compiled from libvc1_b200/csrc/vc1cu_tune.cuh)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "libvc1_b200", "csrc")

MAIN = r"""
#include "vc1cu_tune.cuh"
#include <cstdio>
using namespace vc1cu;
static int bad = 0;
static void check(bool ok, const char* what) { if (!ok) { std::printf("%s\n", what); bad = 1; } }
int main() {
    typedef std::vector<TunePass> L;
    auto key = [](const L& l, int kind = 9, int range = 32) { return tune_key(range, 32, 0, kind, l); };
    const TunePass p{1920, 1080, 0, 0}, cif{352, 288, 0, 0};
    const L one{p}, two{p, p}, uneven{p, cif}, turned{cif, p}, other{p, {640, 360, 0, 0}}, half{{1920, 1080, 2, 0}},
        intra{{1920, 1080, 0, 1}};
    check(key(one) == key(one), "equal launches share a key");
    check(key(one) != key(two), "the number of passes is part of the key");
    check(key(uneven) == key(turned), "the order of the passes is not");
    check(key(uneven) != key(other), "every raster is part of the key, not the first alone");
    check(key(one) != key(half) && key(one) != key(intra), "the MV modes and P-intra are part of the key");
    check(key(one) != key(one, 10) && key(one) != key(one, 9, 64), "so are the instantiation and the ranges");
    // shapes 0 .. 2; two launches under key a: the first is fastest with 0, the second with 1, both
    // together with 1; shape 2 would be best but does not fit the second
    const std::vector<int> a{1}, b{2}, c{3};
    const auto best = tune_choice({{a, {3.0, 3.5, 1.0}}, {b, {2.0, 1.0, 5.0}}, {a, {4.0, 2.0, -1.0}}, {c, {-1.0, -1.0, -1.0}}});
    check(best.at(a) == 1 && best.at(b) == 1 && best.at(c) == -1, "launches that share a key take one shape, the best for both");
    return bad;
}
"""


def test_tuned_shapes_belong_to_their_launches(tmp_path):
    src = tmp_path / "tune.cpp"
    src.write_text(MAIN)
    exe = str(tmp_path / "tune")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
