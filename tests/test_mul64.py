"""The double product on the integer pipes that the plate flexure's transform uses (csrc/cg_mul64.cuh),
checked on the CPU against the hardware's, bit for bit: ties, roundings that carry, signed zeros, the
smallest values it takes, and the values it must refuse."""
import os
import subprocess
import tempfile

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include "cg_mul64.cuh"
int main() {
    double x, w;
    while (std::scanf("%la %la", &x, &w) == 2) {
        if (!cg::plain_value(x)) { std::puts("2"); continue; }
        std::puts(cg::fp_bits(cg::product(cg::Value(x), cg::Weight(w))) == cg::fp_bits(x * w) ? "1" : "0");
    }
}
"""


def run(cases):
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "h.cpp"), os.path.join(d, "h")
        with open(src, "w") as f:
            f.write(HARNESS)
        subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I",
                               os.path.join(ROOT, "cartogenesis_gb300", "csrc"), src, "-o", exe])
        text = "\n".join(f"{float(x).hex()} {float(w).hex()}" for x, w in cases)
        return subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()


def test_product_is_the_hardwares():
    rng = np.random.default_rng(3)
    cases = [(s * x, w) for s in (1.0, -1.0) for x in (0.0, 1.0, 2.0**-967, 1.7976931348623157e308, 2.0 - 2.0**-52)
             for w in (0.0, -0.0, 1.0, -1.0, 1.0 - 2.0**-53, 2.0**-54, np.cos(np.pi / 2))]
    for _ in range(20000):
        short = int(rng.integers(1, 54))   # significands of a few bits tie; of many ones, carry
        x = np.ldexp(float(rng.integers(1, 1 << short) if rng.random() < 0.5 else (1 << short) - 1), int(rng.integers(-900, 900)))
        w = min(1.0, np.ldexp(float(rng.integers(1 << 25, 1 << 26) if rng.random() < 0.5 else (1 << 53) - 1), int(rng.integers(-79, -25))))
        cases.append((x * rng.choice([-1.0, 1.0]), w if w >= 2.0**-54 else 2.0**-54))
    assert set(run(cases)) == {"1"}


def test_other_operands_are_refused():
    assert set(run([(x, 0.5) for x in (5e-324, 2.0**-1022, 2.0**-968, -1e-300, np.inf, -np.inf, np.nan)])) == {"2"}
