"""The tensor-core Tip5 MDS and DFTs restated on the CPU: the byte matrices, the bound on
the 32-bit accumulators and the limb-by-limb recombination (tip5_mma.cuh,
lde_mma.cu, mma8_recombine in mma_i8.cuh) against exact integer arithmetic.  The GPU tests
check the same kernels through whole permutations against the oracle."""
import os
import random
import re

from conftest import ROOT

P = 2**64 - 2**32 + 1
M32 = 2**32
CSRC = os.path.join(ROOT, "triton-vm-prover_b200", "csrc")


def _params():
    src = open(os.path.join(CSRC, "tip5_params.h")).read()
    rc = [int(x, 16) for x in re.findall(r"0x([0-9A-F]+)ull", src)]
    col = re.search(r"TVMC_T5_MDS_FIRST_COLUMN\s*\\?\s*([\d,\s\\]+)", src).group(1)
    mds = [int(x) for x in re.findall(r"\d+", col)]
    assert len(rc) == 80 and len(mds) == 16
    return rc, mds


def weights(m):
    """The eight weights m * 2^(8b) (mod p) as t5m_init forms them in 64 bits."""
    w = [(m << (8 * b)) % 2**64 for b in range(7)]
    return w + [((m << 56) % 2**64 + (m >> 8) * 0xFFFFFFFF) % 2**64]


def recombine(d):
    """mma8_recombine on 32-bit limbs, every intermediate checked to fit."""
    p0, p1, p2, p3 = (d[2 * i] + (d[2 * i + 1] << 8) for i in range(4))
    a = p2 + (p1 >> 16)
    assert max(p0, p1, p2, p3, a) < M32
    s = p0 + (p1 << 16) % M32
    l0, c = s % M32, s >> 32
    s = a + (p3 << 16) % M32 + c
    l1, c = s % M32, s >> 32
    n0 = (p3 >> 16) + 1 + c
    n1 = -n0 % M32
    x = l0 - n0
    l0, b = x % M32, int(x < 0)
    x = l1 - n1 - b
    l1, b = x % M32, int(x < 0)
    m = -b % M32
    x = l0 - m
    l0, b = x % M32, int(x < 0)
    return l0 + ((l1 - b) % M32 << 32)


def test_weights_are_the_products_mod_p_and_accumulators_fit():
    rc, mds = _params()
    for m in mds:
        for b, w in enumerate(weights(m)):
            assert w < 2**64 and (w - (m << (8 * b))) % P == 0
    for t in range(8):
        worst = 255 * sum((w >> (8 * t)) & 255 for m in mds for w in weights(m)) + 255
        assert worst < 2**22


def test_recombined_words_are_canonical_and_exact():
    rc, mds = _params()
    rng = random.Random(5)
    W = [weights(m) for m in mds]
    edge = [0, 1, 2**32 - 1, 2**32, P - 1, P, 2**64 - 1, 0xFF00000000000000, 0x00FF00FF00FF00FF]
    for it in range(400):
        s = [rng.choice(edge) if it < 200 else rng.randrange(2**64) for _ in range(16)]
        if it < len(edge):
            s = [edge[it]] * 16
        k = rng.randrange(80) if it else 0
        r = k % 16
        add = rc[k] * 2**64 % P
        d = [(add >> (8 * t)) & 255 for t in range(8)]
        for c in range(16):
            for b in range(8):
                x = (s[c] >> (8 * b)) & 255
                for t in range(8):
                    d[t] += x * ((W[(r - c) % 16][b] >> (8 * t)) & 255)
        want = (add + sum(mds[(r - c) % 16] * s[c] for c in range(16))) % P
        assert recombine(d) == want


def test_recombination_of_extreme_accumulators():
    top = 2**22 - 1
    rng = random.Random(6)
    cases = [[0] * 8, [top] * 8] + [[rng.choice((0, 1, 255, 256, top)) for _ in range(8)] for _ in range(3000)]
    for d in cases:
        assert recombine(d) == sum(x << (8 * t) for t, x in enumerate(d)) % P


def pow2_mod(e):
    """lde_mma.cu's 2^e (mod p), 0 <= e < 192."""
    s = e - 96 if e >= 96 else e
    v = 1 << s if s < 64 else (1 << (s - 32)) - (1 << (s - 64))
    return P - v if e >= 96 else v


def test_dft_weights_and_accumulator_bounds():
    """B[8k + t][8j + b] = byte t of w_R^(jk) 2^(8b): exact powers of two, and no
    accumulator or partial sum of the recombination can pass 32 bits."""
    for R in (16, 32):
        e1 = 78 * (32 // R)
        assert pow(2, e1, P) == pow(7, (P - 1) // R, P)
        worst = [0] * 8
        for k in range(R):
            d = [0] * 8
            for j in range(R):
                for b in range(8):
                    w = pow2_mod((e1 * j * k + 8 * b) % 192)
                    assert w < P and (w - pow(2, e1 * j * k + 8 * b, P)) % P == 0
                    for t in range(8):
                        d[t] += 255 * ((w >> (8 * t)) & 255)
            worst = [max(x, y) for x, y in zip(worst, d)]
        assert max(worst) < 2**24
        p = [worst[2 * i] + 256 * worst[2 * i + 1] for i in range(4)]
        assert max(p) < M32 and p[2] + (p[1] >> 16) < M32


def test_radix_32_dft_of_bytes_is_the_dft():
    rng = random.Random(7)
    R = 32
    w = pow(7, (P - 1) // R, P)
    x = [rng.choice((0, 2**64 - 1, P, rng.randrange(2**64))) for _ in range(R)]
    for k in (0, 1, 5, 31):
        d = [0] * 8
        for j in range(R):
            for b in range(8):
                v = pow2_mod((78 * j * k + 8 * b) % 192)
                for t in range(8):
                    d[t] += ((x[j] >> (8 * b)) & 255) * ((v >> (8 * t)) & 255)
        assert recombine(d) == sum(x[j] * pow(w, j * k, P) for j in range(R)) % P
