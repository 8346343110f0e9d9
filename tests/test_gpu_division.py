"""The branch-free FP64 divisions and square roots (csrc/bh_div.cuh) against
CUDA's own, bit for bit: random operands over the claimed range (any
significand, few bits, next to powers of two and to all ones, zero numerators
of both signs), and the divisors and arguments whose reciprocals and roots lie
closest to a midpoint of two doubles, where a refinement that is not exact
enough would round the other way."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(REPO, "black-hole-simulator_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
CHECKS = ("rcp_any", "div_by", "sqrt_rn", "1/sqrt", "1/(1/om)", "om^2", "1/xi^3", "h/x near alpha^2")

# prime factors of 2^k + r: a divisor B with an odd 54-bit cofactor C has
# 1 / B = C 2^-k (1 +- 2^-k), next to the midpoint C 2^-k
FACTORS = {
    (100, -1): (3, 5, 5, 5, 11, 31, 41, 101, 251, 601, 1801, 4051, 8101, 268501),
    (102, -1): (3, 3, 7, 103, 307, 2143, 2857, 6529, 11119, 43691, 131071),
    (104, -1): (3, 5, 17, 53, 157, 1613, 2731, 8191, 858001, 308761441),
    (105, -1): (7, 7, 31, 71, 127, 151, 337, 29191, 106681, 122921, 152041),
    (106, -1): (3, 107, 6361, 69431, 20394401, 28059810762433),
    (105, 1): (3, 3, 11, 43, 211, 281, 331, 5419, 86171, 664441, 1564921),
}


def hard_divisors():
    out = set()
    for (k, r), primes in FACTORS.items():
        n = 2 ** k + r
        divisors = {1}
        left = n
        for p in primes:
            assert left % p == 0, (k, r, p)
            left //= p
            divisors |= {d * p for d in divisors}
        assert left == 1, (k, r)
        out |= {b for b in divisors if (n // b).bit_length() == 54 and b.bit_length() <= 53}
    return sorted(out)


def hard_roots():
    """x in [1, 4) with 53 bits whose root lies next to a midpoint m (54 bits,
    odd): m^2 = x + r 2^-106 for a small r (= 1 mod 8), m from r's square
    roots modulo a power of two."""
    out = set()
    for r in range(-4095, 4096):
        if r % 8 != 1:
            continue
        for bits, lo, hi in ((54, 2 ** 106, 2 ** 107), (55, 2 ** 107, 2 ** 108)):
            m = 1
            for b in range(3, bits):                 # m^2 = r modulo 2^(b + 1)
                if (m * m - r) >> b & 1:
                    m += 1 << (b - 1)
            assert (m * m - r) % 2 ** bits == 0
            for q in (m, -m, m + 2 ** (bits - 1), -m + 2 ** (bits - 1)):
                q %= 2 ** bits
                for q in (q, q + 2 ** bits):
                    if lo <= q * q < hi and 2 ** 53 <= q < 2 ** 54:
                        out.add((q * q - r) / 2 ** 106)   # exact: 53 bits
    return sorted(out)


@pytest.fixture(scope="module", params=["--fmad=false", "--fmad=true"])
def lib(request, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("divcheck") / "divcheck.so")
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", request.param,
                        "-Xcompiler", "-fPIC", "-shared", "-I" + CSRC, os.path.join(HERE, "divcheck", "divcheck.cu"),
                        "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(so)
    L.divcheck_random.argtypes = [C.c_int64, C.c_uint64, C.c_void_p, C.c_void_p]
    for f in (L.divcheck_list, L.divcheck_roots):
        f.argtypes = [C.c_void_p, C.c_int, C.c_uint64, C.c_void_p, C.c_void_p]
    assert L.divcheck_checks() == len(CHECKS)
    return L


def run(call):
    import torch
    count = torch.zeros(len(CHECKS), dtype=torch.int64, device="cuda")
    first = torch.zeros((len(CHECKS), 2), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert call(C.c_void_p(count.data_ptr()), C.c_void_p(first.data_ptr())) == 0
    bad = {c: (int(k), [float(x).hex() for x in f])
           for c, k, f in zip(CHECKS, count.cpu().numpy(), first.cpu().numpy()) if k}
    assert not bad, bad


@pytest.mark.parametrize("seed", [1, 2])
def test_random_operands(lib, seed):
    run(lambda c, f: lib.divcheck_random(1 << 26, seed, c, f))


@pytest.mark.parametrize("what", ["reciprocals", "roots"])
def test_next_to_midpoints(lib, what):
    import torch
    x, f = (hard_divisors(), lib.divcheck_list) if what == "reciprocals" else (hard_roots(), lib.divcheck_roots)
    assert len(x) > 100
    t = torch.tensor([float(v) for v in x], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    run(lambda c, first: f(C.c_void_p(t.data_ptr()), len(x), 3, c, first))
