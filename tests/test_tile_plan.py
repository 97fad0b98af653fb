"""The division of the tile kernels' work into units: the best one, found in few tries."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include "rayleighchebyshevgpgpu_b200/csrc/rc_tileplan.h"
static int one_by_one(int nz, int64_t columns, int64_t ctas) {
    double best = 1e300;
    int planes = 0;
    for (int k = 1; k <= nz; ++k) {
        const int ml = (nz + k - 1) / k;
        const int64_t units = columns * ((nz + ml - 1) / ml);
        const double cost = (double)((units + ctas - 1) / ctas) * (ml + 1.2);
        if (cost < best) { best = cost; planes = ml; }
        if (ml <= 4) break;
    }
    return planes;
}
int main() {
    const int ctas[] = {148, 147, 144, 140, 132, 37, 1};
    int most = 0;
    std::srand(1);
    for (int t = 0; t < 60000; ++t) {
        const int nz = (int)std::exp(std::rand() / (double)RAND_MAX * std::log(4000.0));
        const int64_t columns = (int64_t)std::exp(std::rand() / (double)RAND_MAX * std::log(5000.0));
        const int64_t c = ctas[std::rand() % 7];
        int tries = 0;
        if (rcb::tile_planes(nz, columns, c, nullptr, &tries) != one_by_one(nz, columns, c)) {
            std::printf("nz %d columns %lld ctas %lld\n", nz, (long long)columns, (long long)c);
            return 1;
        }
        most = tries > most ? tries : most;
    }
    for (int nz : {12000, 100000, 1000000})
        for (int64_t columns : {1, 2, 4, 40}) {
            int tries = 0;
            rcb::tile_planes(nz, columns, 148, nullptr, &tries);
            most = tries > most ? tries : most;
        }
    std::printf("%d\n", most);
    return most > 100;
}
"""


def test_units_are_the_best_and_found_quickly(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", ROOT, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
