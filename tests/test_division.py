"""The divisions by a known divisor of csrc/kernels/device_utils.cuh against the IEEE quotient, on the CPU: the functions
themselves, compiled for the host."""
import subprocess

from shield_sisa_b200 import build

SOURCE = r"""
#include "device_utils.cuh"
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

static float value(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
static uint32_t bits(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }

// prints the largest x of [lo, hi) whose result is not the quotient's, as bits (0: none), and the most steps between the two
template <typename F> static void sweep(uint32_t lo, uint32_t hi, float d, F divide) {
    std::atomic<uint32_t> top{0}, steps{0};
    const auto raise = [](std::atomic<uint32_t>& a, uint32_t v) { uint32_t o = a.load(); while (o < v && !a.compare_exchange_weak(o, v)) {} };
    std::vector<std::thread> threads;
    for (uint32_t t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            uint32_t mine = 0, most = 0;
            for (uint64_t b = uint64_t(lo) + t; b < hi; b += 8) {
                const uint32_t got = bits(divide(value(uint32_t(b)))), want = bits(value(uint32_t(b)) / d);
                if (got == want) continue;
                mine = uint32_t(b);
                const uint32_t off = uint32_t(std::labs(long(got) - long(want)));
                if (off > most) most = off;
            }
            raise(top, mine);
            raise(steps, most);
        });
    for (std::thread& t : threads) t.join();
    printf("%u %u\n", top.load(), steps.load());
}

int main() {
    sweep(0, 0x7f800001u, 6.0f, [](float x) { return sb::div6(x); });                       // zero, all positive numbers, infinity
    const float root = 1.41421356f;
    sweep(0, 0x7f800001u, root, [=](float x) { return sb::div_known(x, root, 1.0f / root); });
    // other divisors: both ends of the range, its binades' ends, and some between; all mantissas, at 1, 2^-102 and 2^126
    std::vector<uint32_t> ds = {0x3f800000u, 0x3f800001u, 0x3fffffffu, 0x40000001u, 0x407fffffu, 0x40800001u, 0x40ffffffu, 0x417fffffu};
    for (uint32_t i = 0; i < 8; ++i) ds.push_back(0x3f800000u + (2654435761u * (i + 1) & 0x1ffffffu));
    for (uint32_t b : ds) {
        const float d = value(b), z = 1.0f / d;
        for (uint32_t e : {127u, 25u, 253u}) sweep(e << 23, (e + 1) << 23, d, [=](float x) { return sb::div_known(x, d, z); });
    }
}
"""


def test_divisions_by_known_divisors_give_the_quotients_bits(tmp_path):
    src, exe = tmp_path / "division.cu", tmp_path / "division"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-Xcompiler", "-mfma,-ffp-contract=off", str(src), "-o", str(exe), "-lpthread"], check=True,
                   capture_output=True)
    rows = [[int(v) for v in line.split()] for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 2 + 3 * 16
    assert rows[0] == [(127 - 122) << 23 | 1 << 21, 1]           # 1.25 x 2^-122: the line that div6 states, one step
    assert 0 < rows[1][0] < (127 - 105) << 23 and rows[1][1] == 1   # d = sqrt 2: below 2^-105, one step
    assert all(row == [0, 0] for row in rows[2:])
