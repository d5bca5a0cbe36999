"""The resident PCG's fixed-point sums (lightfem_gb300/csrc/cg_fixed.hpp), run on the host:
a total that is accepted is the exact sum of the shares to the sums' units, whatever the
shares, and one near the last total is accepted.

Bounds, with the scale 2^e <= the last total: a share is rounded to 2^-56 (FP32 pairs)
or 2^-78 (FP64) of the scale, a CTA's FP64 sum to 2^-70, each by half a unit (pairs: a
quarter more for the remainders' own sum); the total to 2^-46 (a pair) or 2^-53 of
itself.
"""

import math
import os
import subprocess

import numpy as np
import pytest

from host_cpp import ROOT

CTAS = (1, 2, 16, 152, 254)
THREADS = {True: (32, 1024), False: (32, 512)}  # mixed: the most a CTA has


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    out = tmp_path_factory.mktemp("sums")
    exe = os.path.join(out, "fixed_sums_check")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-ffp-contract=off",
                    os.path.join(ROOT, "tests", "host", "fixed_sums_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)

    def run(cases):
        src, dst = os.path.join(out, "in.bin"), os.path.join(out, "out.bin")
        with open(src, "wb") as fh:
            fh.write(np.int64(len(cases)).tobytes())
            for mixed, previous, shares in cases:
                fh.write(np.array([mixed, *shares.shape], np.int64).tobytes() + np.float64(previous).tobytes())
                fh.write(np.ascontiguousarray(as_pairs(shares) if mixed else shares).tobytes())
        subprocess.run([exe, src, dst], check=True)
        return np.fromfile(dst).reshape(-1, 4)

    return run


def as_pairs(shares):
    hi = shares.astype(np.float32)
    return np.stack([hi, (shares - hi).astype(np.float32)], -1)


def check(sums, cases):
    results = sums(cases)
    for (mixed, previous, shares), (accepted, overflow, hi, lo) in zip(cases, results):
        assert not overflow
        values = as_pairs(shares).astype(np.float64) if mixed else shares
        exact = math.fsum(values.ravel())
        scale = 2.0 ** math.floor(math.log2(previous))
        if accepted:
            units = 1.25 * 2.0 ** -57 if mixed else 2.0 ** -79
            bound = shares.size * units * scale + 2.0 ** (-46 if mixed else -53) * abs(exact)
            if not mixed:
                bound += shares.shape[0] * 2.0 ** -71 * scale
            assert abs(hi + lo - exact) <= bound, (mixed, shares.shape, exact / scale)
        else:
            assert not (2.0 ** -9 <= exact / scale <= 8.0 and np.abs(shares).max() < 8 * scale), (shares.shape,
                                                                                              exact / scale)
    return results[:, 0]


@pytest.mark.parametrize("mixed", [True, False])
def test_random_shares(sums, mixed):
    """Totals from 2^-14 to 2^14 of the last one, shares of one size and of many."""
    rng = np.random.default_rng(7)
    cases = []
    for ctas in CTAS:
        for threads in THREADS[mixed]:
            for _ in range(12):
                s = rng.standard_normal((ctas, threads)) ** 2 * np.exp(rng.uniform(0, 4) * rng.standard_normal((ctas, threads)))
                if rng.random() < 0.3:
                    s[rng.random(s.shape) < 0.4] *= -1e-3
                last = 2.0 ** rng.uniform(-60, 60)
                cases.append((mixed, last, s * (last * 2.0 ** rng.uniform(-14, 14) / s.sum())))
    accepted = check(sums, cases)
    assert 0.3 < accepted.mean() < 0.9  # both ways are met


@pytest.mark.parametrize("mixed", [True, False])
def test_equal_shares_up_to_their_limit(sums, mixed):
    """Every thread's share the same, from far below the last total to the largest share a
    thread may have: sums that run past a limb, a word or 64 bits are not taken for small
    ones (a total of 256 j + 3 scales reads as 3 where 64 bits of 2^-56 wrap)."""
    cases = []
    for ctas in CTAS:
        for threads in THREADS[mixed]:
            n = ctas * threads
            totals = [2.0 ** k for k in range(-11, 22)] + [256.0 * j + 3 for j in (1, 2, 5, 40, 127)]
            for total in totals + [ctas * t for t in totals]:
                cases.append((mixed, 1.0, np.full((ctas, threads), total / n)))
            top = 32.0 if mixed else 512.0
            cases += [(mixed, 1.0, np.full((ctas, threads), float(s * f))) for s in (1, -1)
                      for f in (float(np.nextafter(np.float32(top), np.float32(0))), top / 2, top, 4 * top)]
    check(sums, cases)
