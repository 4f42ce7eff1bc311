"""Which pressure solves may be in flight together (csrc/coop_share.cuh): every admitted set of launches
has a place for each block wherever the blocks that share SMs lie, a launch alone is always admitted, and
launches of the sharing kind are admitted up to the whole GPU."""
import subprocess

from banana_b200 import build as bld

_PROGRAM = r"""
#include "coop_share.cuh"
#include <cstdio>
using namespace bnn;
int main() {
    const int numSM = 5;
    std::vector<CoopLoad> kinds;
    for(int w = 1; w <= numSM; ++w) kinds.push_back({w, 0, 0});
    for(int per = 1; per <= 3; ++per)
        for(int b = 1; b <= per * numSM; ++b) kinds.push_back({0, b, b * (kShareUnits / per)});
    for(const CoopLoad& l : kinds)
        if(!coop_fits(l, numSM)) { std::printf("a launch alone is refused\n"); return 1; }
    int admitted = 0;
    for(const CoopLoad& a : kinds)
        for(const CoopLoad& b : kinds)
            for(const CoopLoad& c : kinds) {
                if(!coop_fits(a + b, numSM) || !coop_fits(a + b + c, numSM)) continue;
                ++admitted;
                const CoopLoad all = a + b + c;
                // the sharing blocks on as many SMs as they can reach: the others need the rest
                if(all.whole > numSM - (all.blocks < numSM ? all.blocks : numSM)) { std::printf("no empty SM left\n"); return 1; }
                if(all.shared > (numSM - all.whole) * kShareUnits) { std::printf("no room to share\n"); return 1; }
            }
    const CoopLoad third{0, numSM, numSM * (kShareUnits / 3)};
    if(!coop_fits(third + third + third, numSM) || coop_fits(third + third + third + third, numSM)) {
        std::printf("three thirds\n");
        return 1;
    }
    std::printf("ok %d\n", admitted);
    return 0;
}
"""


def test_admitted_launches_all_find_a_place(tmp_path):
    src = tmp_path / "share.cpp"
    src.write_text("#include <vector>\n" + _PROGRAM)
    exe = tmp_path / "share"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(bld.CSRC), "-o", str(exe), str(src)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
