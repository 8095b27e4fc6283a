"""The tensor-core rounds' arithmetic on the CPU: the digit matrices, the bound of
the sums, and the inline PTX of era-boojum-cuda_b200/csrc/tc.cuh."""
import os
import random

import pytest

import ptx_model as pm

HERE = os.path.dirname(os.path.abspath(__file__))
TC = os.path.join(HERE, "..", "era-boojum-cuda_b200", "csrc", "tc.cuh")
P = (1 << 64) - (1 << 32) + 1
EPS = (1 << 32) - 1
M32, M64 = (1 << 32) - 1, (1 << 64) - 1
BLOCKS = pm.asm_blocks(TC)
EDGE = [0, 1, EPS, 1 << 32, P - 2, P - 1, P, P + 1, 1 << 63, M64 - EPS, M64 - 1, M64, 0xFFFFFFFEFFFFFFFF]


def fold(d):
    """fold_digits: the C++ around its asm block, restated."""
    p = [d[2 * i] + (d[2 * i + 1] << 8) for i in range(4)]
    assert max(p) <= M32
    l, h = p[0] + (p[1] << 16), p[2] + (p[3] << 16)
    t = l + (h >> 32) * EPS
    assert t < 1 << 50  # so that the carry's EPS cannot carry again
    return pm.run(BLOCKS[("fold_digits", 0)], [t, h & M32])


def test_fold_digits():
    rnd = random.Random(1)
    top = 256 * 255 * 255  # 32 words a row
    cases = [[top] * 8, [128 * 255 * 255] * 8, [0] * 8, [0] * 4 + [255] * 4, [255] * 8, [0] * 4 + [255, 255, 255, 256]]
    cases += [[rnd.choice((0, 1, 255, 256, top, rnd.randint(0, top))) for _ in range(8)] for _ in range(4000)]
    for d in cases:
        got = fold(d)
        assert got <= M64 and got % P == sum(v << (8 * j) for j, v in enumerate(d)) % P, d


def test_mul():
    rnd = random.Random(2)
    vals = EDGE + [rnd.getrandbits(64) for _ in range(60)]
    for a in vals:
        for b in vals:
            q = a * b
            lo, hi = q & M64, q >> 64
            z = (hi & M32) * EPS + (lo & M32)
            assert z <= M64
            got = pm.run(BLOCKS[("mul", 0)], [z, lo >> 32, hi >> 32])
            assert got % P == q % P, (a, b)


@pytest.mark.parametrize("points,root", [(16, pow(2, 156, P)), (32, pow(2, 78, P))])
def test_digit_matrix(points, root):
    """Bytes in, 8-bit digits of the matrix entries, sums exact in 32 bits (16 points: below fold_digits' bound)."""
    assert root == pow(7, (P - 1) // points, P)
    rnd = random.Random(points)
    bits = points.bit_length() - 1
    brev = [int(format(o, f"0{bits}b")[::-1], 2) for o in range(points)]
    x = [rnd.choice((M64, rnd.getrandbits(64))) for _ in range(points)]
    for o in (0, 1, points // 2, points - 1):
        m = [pow(root, i * brev[o], P) for i in range(points)]
        d = [0] * 8
        for i in range(points):
            for b in range(8):
                entry = m[i] * pow(2, 8 * b, P) % P
                for j in range(8):
                    d[j] += (entry >> (8 * j) & 255) * (x[i] >> (8 * b) & 255)
        assert max(d) <= 8 * points * 255 * 255 < 1 << (20 + bits)
        assert fold(d) % P == sum(a * b for a, b in zip(m, x)) % P
