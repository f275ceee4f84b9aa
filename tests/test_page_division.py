"""CPU: the division of a token's index by the page size in FP8 decode on pairs of SMs (`reciprocal` and `page_of_token`,
csrc/attn_shared.cuh), restated here, against integer division."""
import os
import random
import re
import subprocess

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashmla_b200", "csrc", "attn_shared.cuh")


def test_page_of_a_token():
    text = open(SOURCE).read()
    assert re.search(r"mul = \(uint32_t\)\(\(\(uint64_t\)1 << \(31 \+ l\)\) / \(uint64_t\)d \+ 1\);\s*shift = 31 \+ l;", text)
    assert "(uint32_t)(((uint64_t)id * p.pbs_mul[scope]) >> p.pbs_shift[scope])" in text
    rng = random.Random(3)
    sizes = list(range(1, 700)) + [2 ** k + e for k in range(10, 31) for e in (-1, 0, 1)] + [2 ** 31 - 1]
    for d in sizes:
        l = (d - 1).bit_length()
        mul, shift = (1 << (31 + l)) // d + 1, 31 + l
        assert mul < 2 ** 32 and shift < 64
        last = 2 ** 31 - 1
        edges = [0, 1, d - 1, d, d + 1, last, last - 1] + [k * d + e for k in (last // d, last // d - 1, last // (2 * d)) for e in (-1, 0, 1)]
        for n in edges + [rng.randrange(2 ** 31) for _ in range(40)]:
            if 0 <= n <= last:
                assert n * mul < 2 ** 64 and n * mul >> shift == n // d, (n, d)


def test_the_functions_of_the_source(tmp_path):
    """`reciprocal` and `page_of_token` themselves, compiled for the host."""
    text = open(SOURCE).read()
    take = lambda start: text[text.index(start):text.index("\n}\n", text.index(start)) + 3]
    program = """
#include <cstdint>
#include <cstdio>
#define __device__
#define __forceinline__ inline
struct Params { int pbs[2]; uint32_t pbs_mul[2]; int pbs_shift[2]; };
""" + take("__device__ __forceinline__ uint32_t page_of_token(") + take("static void reciprocal(") + """
int main() {
    int d; unsigned n, wrong = 0, seen = 0;
    while (std::scanf("%d %u", &d, &n) == 2) {
        Params p = {};
        uint32_t off;
        p.pbs[1] = d;
        reciprocal(d, p.pbs_mul[1], p.pbs_shift[1]);
        ++seen;
        if (page_of_token(p, 1, n, off) != n / d || off != n % d) ++wrong;
    }
    std::printf("%u %u", wrong, seen);
}
"""
    (tmp_path / "division.cpp").write_text(program)
    subprocess.run(["g++", "-O1", "-o", tmp_path / "division", tmp_path / "division.cpp"], check=True)
    rng, last = random.Random(7), 2 ** 31 - 1
    sizes = list(range(1, 700)) + [2 ** k + e for k in range(10, 31) for e in (-1, 0, 1)] + [last]
    pairs = [(d, n) for d in sizes for n in [0, d - 1, d, last, last // d * d, last // d * d - 1] + [rng.randrange(2 ** 31) for _ in range(20)] if 0 <= n <= last]
    out = subprocess.run([tmp_path / "division"], input="\n".join("%d %d" % p for p in pairs), capture_output=True, text=True, check=True).stdout
    assert out.split() == ["0", str(len(pairs))]
