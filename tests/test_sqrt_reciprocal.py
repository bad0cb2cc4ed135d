"""The Cholesky pivots' square root and reciprocal (csrc/sqrt_reciprocal.h) against
sqrt(d) and 1.0 / s, both correctly rounded in IEEE arithmetic.

The final steps are exact to 2^-103 before rounding, so beside random and edge
mantissas the points that lie nearest to a rounding boundary are enumerated:
  - roots: all d whose root is within 2^-96 of a boundary m, an odd multiple of
    half a unit: m^2 = c mod 2^54 (or 2^55), |c| < 2^11, solved bit by bit
  - reciprocals: all s with |s m - 2^106| <= 16 for an odd m, from the divisors
    of 2^106 + c (HARD_S below, found with a factorisation of each of them)
The starting value is the rounded FP32 reciprocal root, moved by up to two units:
the error CUDA documents for rsqrtf."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "gmgs-3d_gb300" / "csrc"

HARD_S = """
1014ca35e947b6 1024a3bd98da02 10699d36aec84e 109107683ee29e 10aadc6f562fdc 10ad803397a510 10af911aa26396
10d03f8a57cc76 10ed85c351e224 110af85de838ce 110d10000221a2 1125e52b034982 113deff6b41e35 115efb8b10aa42
11d3799c32581e 11f98ea5d9b262 120a8f5bbf2106 122aea483b4410 12492492492490 124936db76db70 12563fca7b8530
12565220c47ad0 1292074009a630 12af4d6bc06922 12bf5907e316d2 12d2d2d2d2d2d4 12e3c6a0509ca4 12e93952a2ed6e
130117cb1c0d50 130a0dd90e13a2 1320bffffb37d0 1320c99064c830 132160ccc0848c 134d8fe343ef42 13541c0067f83c
1379cb88f092f2 1387bffffb1e10 13a324a526d5ee 13a7a1d01d1ec2 13d75d54b37492 1403e897077b16 142f1a2b6c8e90
14873ecade304c 14a6fb45f5d782 14cad5a5fa03ee 1520e032e63b90 15555555555554 155f2490c86132 156a8cb0234262
159aa11aaecb86 16026c81a85766 161c2909f39d4b 163baaac17d1e2 163dd0554d0122 16d6422e5cf246 16f0f27bf434d6
16fae7ba173812 172f10bf899124 1733e76d85fcd0 17641c46f799ee 178cb7d5d6e322 178d42e524dcdc 179376969ecfd0
17f52093014f0e 1806c89fcb9452 181efe51ead722 18387f2dc43370 18401cbcdb5596 184a12efef626e 1860cbb1b40ef0
1860e4128bf110 186f1e976d35b0 18f2b1225b0d70 190dcff22c6050 191c4c8e264710 1943ecc40c6590 194ab05a4ecedc
194c4511fa3124 195608aa510030 195615554effd0 1960a45d1a71e6 198049c39bbe50 1999998cccccd0 199d2b42ffe9f4
199e1b447e99c2 19cd0026800cd0 19f142d24e1352 1a0b8ffffcbe8e 1a149bad85de72 1a2ce4d7478a06 1a6f41dab98cb2
1aa7c88ee59082 1ae6849e786ad2 1b227794e85702 1bea3278b789d2 1c2693dcf34742 1c36899addce3c 1c384d119331c4
1c4d3aabd478f6 1c69bf28eba166 1c928b5b9dc714 1d5b9032f086be 1d650c90101950 1da210daeb138e 1de441d5331432
1de4a0d00fa9b2 1e20adbc4078a2 1e756f08df1792 1e8d517d09c5c2 1e9a9473949bf6 1ee13ffff847b0 1ef43974550f69
1ef7930608393e 1f65fad23b0d86 1f739bd459bea2 1fa01f23c0c510 1fcea3254679b0 1fe24bffeb8794 1ffb8a8b628dbc
1ffffff8000001 1ffffffffffffd 1fffffffffffff
"""

PROGRAM = r"""
#include "sqrt_reciprocal.h"
#include <cstdio>
#include <cstdlib>
#include <random>
static long bad = 0, count = 0;
static void check(double d) {
    const double root = std::sqrt(d), inverse = 1.0 / root;
    for (int k = -2; k <= 2; ++k) {
        float y = (float)(1.0 / root);
        for (int i = 0; i < std::abs(k); ++i) y = std::nextafterf(y, k > 0 ? 4.f : 0.f);
        double s, r;
        gmgs::sqrt_reciprocal(d, y, s, r);
        ++count;
        if ((s != root || r != inverse) && bad++ < 10) std::printf("%a from %a: %a %a, not %a %a\n", d, y, s, r, root, inverse);
    }
}
int main(int, char** argv) {
    std::mt19937_64 g(1);
    for (int i = 0; i < 2000000; ++i) check(std::ldexp((double)(g() >> 11 | 1ull << 52), (int)(g() % 241) - 120 - 52));
    for (int e = -120; e <= 120; ++e)                       // around powers of two: all-ones mantissas, 1 + a few units
        for (int k = -40; k <= 40; ++k) check(std::ldexp(1.0 + k * (k < 0 ? 0x1p-53 : 0x1p-52), e));
    for (int k = 0; k < 100000; ++k) {                      // roots near 1 and near 2
        check((1.0 + k * 0x1p-52) * (1.0 + k * 0x1p-52));
        check((2.0 - k * 0x1p-52) * (2.0 - k * 0x1p-52));
    }
    for (int64_t c = 1 - 2048; c < 2048; c += 8) {          // odd squares are 1 modulo 8
        uint64_t x = 1;
        for (int b = 3; b < 56; ++b)
            if ((x * x - (uint64_t)c) >> b & 1) x += 1ull << (b - 1);
        for (int n = 54; n <= 55; ++n)
            for (int v = 0; v < 4; ++v) {
                const uint64_t m = ((v & 1 ? 0 - x : x) + (v & 2 ? 1ull << (n - 1) : 0)) & ((1ull << n) - 1);
                if (m >> 53 != 1) continue;                 // 2^53 <= m < 2^54
                const unsigned __int128 d = (unsigned __int128)m * m - (__int128)c;
                if ((d >> 107 ? 55 : 54) != n || (uint64_t)d & ((1ull << n) - 1)) continue;
                check(std::ldexp((double)(uint64_t)(d >> n), n - 106));
            }
    }
    const long before = count;
    for (char* p = argv[1]; *p;) {
        const double s = std::ldexp((double)std::strtoull(p, &p, 16), -52);
        double d = s * s;
        for (int i = 0; i < 6; ++i) d = std::nextafter(d, 0.0);
        for (int i = 0; i < 12; ++i, d = std::nextafter(d, 8.0)) check(d);
        while (*p == ' ') ++p;
    }
    std::printf("%ld values, %ld of them around hard reciprocals, %ld wrong\n", count, count - before, bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_both_correctly_rounded(tmp_path):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(PROGRAM)
    build = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC), str(src), "-o", str(exe)],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe), " ".join(HARD_S.split())], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    assert "wrong" in run.stdout and int(run.stdout.split(" values, ")[1].split()[0]) > 5000
