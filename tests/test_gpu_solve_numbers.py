"""The team sums of the solve launches against exactly rounded sums (math.fsum): as accurate as FP64
additions, for every team, and a sum of infinities and NaN what IEEE arithmetic gives. Their divisions
against FP64 ones rounded to float."""
import math
import os
import subprocess

import numpy as np
import pytest
from conftest import ROOT

from bounce_softbody_gb300 import build

pytestmark = pytest.mark.gpu

ROUNDS = 24
TEAMS = [(1, 1, 0), (3, 4, 0), (16, 8, 0), (17, 1, 0), (33, 16, 0), (152, 16, 0), (1, 5, 1), (2, 8, 2), (5, 3, 5),
         (8, 16, 8), (16, 8, 16)]  # CTAs, warps, cluster


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("numbers") / "solve_numbers")
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "solve_numbers.cu"), "-o", exe], check=True)
    return exe


def team_sums(program, team, values):
    ctas, warps, _ = team
    out = subprocess.run([program], input=np.array(team, np.int32).tobytes() + values.tobytes(), stdout=subprocess.PIPE,
                         check=True, timeout=120).stdout
    totals = np.frombuffer(out).reshape(ctas, ROUNDS)
    # every CTA takes its decisions on the same bits
    assert (totals.view(np.uint64) == totals[:1].view(np.uint64)).all()
    return totals[0]


@pytest.mark.parametrize("team", TEAMS)
def test_one_value_keeps_its_bits(program, team):
    """One warp's value among zeros: the sum is that value."""
    ctas, warps, _ = team
    rng = np.random.default_rng(ctas)
    want = np.ldexp(rng.uniform(0.5, 1.0, ROUNDS), rng.integers(-300, 300, ROUNDS)) * rng.choice([-1.0, 1.0], ROUNDS)
    want[:6] = [5e-324, -2.0 ** -1022 * (1 - 2.0 ** -52), np.finfo(float).max, -np.inf, np.nan, 1.0 + 2.0 ** -52]
    v = np.zeros((ctas, warps, ROUNDS))
    v[rng.integers(0, ctas, ROUNDS), rng.integers(0, warps, ROUNDS), np.arange(ROUNDS)] = want
    got = team_sums(program, team, v)
    nan = np.isnan(want)
    assert np.isnan(got[nan]).all() and np.array_equal(got[~nan], want[~nan])


@pytest.mark.parametrize("team", TEAMS)
def test_sums_are_as_accurate_as_fp64_additions(program, team):
    """Terms of all magnitudes. Of a term at least 54 bits below the largest one's first are kept at each of
    three levels (warps, CTAs of a lane, lanes), and the total is rounded once: an error of at most
    3 * 2^-54 of the largest per term (below FP64 additions' 2^-53 per addition and level) and half an
    ulp of the total."""
    ctas, warps, _ = team
    rng = np.random.default_rng(100 + ctas)
    v = rng.standard_normal((ctas, warps, ROUNDS)) * 2.0 ** rng.integers(-40, 1, (ctas, warps, ROUNDS))
    v[..., ROUNDS // 2:] = np.abs(v[..., ROUNDS // 2:])
    got = team_sums(program, team, v)
    for r in range(ROUNDS):
        exact = math.fsum(v[..., r].ravel())
        largest = np.abs(v[..., r]).max()
        # the sums of a level may be larger than their terms
        reach = max(largest, np.abs(v[..., r].sum(1)).max(), abs(exact))
        assert abs(got[r] - exact) <= 3 * 2.0 ** -54 * reach * (ctas * warps - 1) + 0.5 * np.spacing(abs(exact))


@pytest.mark.parametrize("team", [t for t in TEAMS if t[0] * t[1] > 1])
def test_sums_that_are_not_finite(program, team):
    ctas, warps, _ = team
    big = np.finfo(float).max
    pairs = [(np.inf, 1.0, np.inf), (-np.inf, -1e300, -np.inf), (np.inf, -1e300, np.inf), (np.inf, np.inf, np.inf),
             (np.inf, -np.inf, np.nan), (np.nan, np.inf, np.nan), (np.nan, 1.0, np.nan), (big, big, np.inf),
             (-big, -big, -np.inf), (big, -big, 0.0), (big, 2.0 ** 969, big), (big, 2.0 ** 970, np.inf)]
    v = np.zeros((ctas * warps, ROUNDS))
    want = np.zeros(ROUNDS)
    for r, (a, b, c) in enumerate(pairs):
        v[0, r], v[-1, r], want[r] = a, b, c
    got = team_sums(program, team, v)
    assert np.array_equal(got, want, equal_nan=True)


def test_divisions_are_fp64_ones_rounded_to_float(program):
    rng = np.random.default_rng(7)
    n = 1 << 20
    b = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-60, 60, n)) * rng.choice([-1.0, 1.0], n)
    # quotients anywhere
    a = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-60, 60, n))
    # quotients at the midpoint of two floats, to a few units in the last place of a double
    q = rng.uniform(1.0, 2.0, n).astype(np.float32)
    q[: n // 16] = np.float32(1.0)
    q[n // 16: n // 8] = np.nextafter(np.float32(2.0), np.float32(0.0))
    mid = q.astype(np.float64) + 2.0 ** -24 * rng.choice([-1.0, -0.5, 1.0], n)
    near = (mid * b).view(np.int64) + rng.integers(-6, 7, n)
    special = np.array([0.0, -0.0, 1.0, -3.0, 5e-324, 2.0 ** -1022, np.finfo(float).max, np.inf, -np.inf, np.nan, 1e-30,
                        1e30, 2.0 ** 127, 2.0 ** -126, 2.0 ** -149])
    sa, sb = (x.ravel() for x in np.meshgrid(special, special))
    num, den = np.concatenate([a, near.view(np.float64), sa]), np.concatenate([b, b, sb])
    with np.errstate(all="ignore"):
        want = (num / den).astype(np.float32)
    pairs = np.ascontiguousarray(np.stack([num, den], 1))
    out = subprocess.run([program], input=np.array([len(num), 0, -1], np.int32).tobytes() + pairs.tobytes(),
                         stdout=subprocess.PIPE, check=True, timeout=120).stdout
    got = np.frombuffer(out).astype(np.float32)
    nan = np.isnan(want)
    assert np.isnan(got[nan]).all()
    assert np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))
