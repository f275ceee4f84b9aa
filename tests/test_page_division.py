"""CPU: the division of a token's index by the page size in FP8 decode on pairs of SMs (`reciprocal` and `page_of_token`,
csrc/attn_shared.cuh), restated here, against integer division."""
import os
import random
import re

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
