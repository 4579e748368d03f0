"""Values at which an integer-pipe operation or a shortcut of the FP64 step has
to hand over or to keep a sign: the step against the CPU oracle and the
operations, compiled for the host, against IEEE arithmetic, bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import oracle as orc
from sw2_gb300 import cases, lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GXX = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")

PRELUDE = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "sigmath.cuh"
using namespace sw2g;
static uint64_t st = 0x9216D5D98979FB1BULL;
static uint64_t next() {  // SplitMix64
  uint64_t z = (st += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
static double from(uint64_t b) { double d; std::memcpy(&d, &b, 8); return d; }
static uint64_t bits(double d) { uint64_t b; std::memcpy(&b, &d, 8); return b; }
static uint64_t frac() { return next() >> 12; }
"""


def host_run(tmp_path, text, *args):
    c, exe = tmp_path / "h.cpp", tmp_path / "h"
    c.write_text(PRELUDE + text)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-I", str(tmp_path), "-I",
                    os.path.join(ROOT, "sw2_gb300", "csrc"), "-o", str(exe), str(c)], check=True)
    return subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True).stdout.split()


def bitwise(a, b):
    """Equal bit for bit, NaNs as NaNs."""
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan]) and np.array_equal(np.isnan(a), np.isnan(b))


MUL3 = r"""
// c in 2^-902 .. 2^102, |a*c| at most 2^101, b any number a Courant number may
// leave (zeros and subnormals too): where sig_mul3_far does not say so, sig_mul3
// is the rounded product; and it does not for factors and products well inside
int main(int, char** argv) {
  long long wrong = 0, refused = 0, taken = 0;
  for (long long i = 0; i < atoll(argv[1]); i++) {
    const bool wide = next() % 2;
    const int ec = wide ? 121 + next() % 1004 : 874 + next() % 186;
    uint64_t c = ((uint64_t)ec << 52) | frac(), a = ((wide ? 1 + next() % 2046 : 874 + next() % 186) << 52) | frac();
    uint64_t b = ((wide ? next() % 2047 : 874 + next() % 186) << 52) | frac();
    const int k = next() % 16;
    if (k == 0) b = 0;                                   // a Courant number of 1
    if (k == 1) b = bits(1.0 - from(bits(1.0) - 1));     // and next to it
    if (k == 2) a = frac();                              // subnormal
    if (k == 3) a = 0x7ff0000000000000ULL | (next() % 2);  // inf, NaN
    if (k == 4) a = ((uint64_t)(2147 - ec > 2046 ? 2046 : 2147 - ec) << 52) | frac(), b = next() % 2 ? 0 : frac();
    if (k != 3 && (int)(a >> 52) + ec > 2147) continue;
    const bool far = sig_mul3_far(a >> 32, b >> 32, c >> 32);
    if (!far) {
      taken++;
      wrong += sig_mul3(a, b, c) != bits(from(a) * from(b) * from(c));
    }
    bool inside = true;
    const uint64_t x[3] = {a, b, c};
    for (uint64_t v : x) inside = inside && (v >> 52) >= 874 && (v >> 52) < 1060;
    refused += inside && far;
  }
  printf("%lld %lld %d\n", wrong, refused, taken > 100000);
}
"""


@GXX
def test_three_factor_products_match_ieee_or_are_refused(tmp_path):
    assert host_run(tmp_path, MUL3, 5_000_000) == ["0", "0", "1"]


DIV = r"""
int main(int, char** argv) {
  long long wrong = 0;
  for (long long i = 0; i < atoll(argv[1]); i++) {
    uint64_t a = 0x3ff0000000000000ULL | frac(), b = 0x3ff0000000000000ULL | frac();
    switch (next() % 8) {
      case 0: b |= ((1ULL << 23) - 1) << 29; break;             // leading bits that round up to 2
      case 1: b &= ~(((1ULL << 23) - 1) << 29); break;          // and to the least above 1
      case 2: b = 0x3fffffffffffffffULL - next() % 64; break;
      case 3: b = 0x3ff0000000000000ULL + next() % 64; break;
      case 4: a = bits(from(b) * (from(a) + std::ldexp((double)(next() % 8 + 1), -54))); break;  // next to a midpoint
      case 5: a = 0x3fffffffffffffffULL - next() % 64; break;
      default: break;
    }
    wrong += sig_div(a, b) != bits(from(a) / from(b));
  }
  printf("%lld\n", wrong);
}
"""


@GXX
@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_quotients_hold_with_a_reciprocal_one_ulp_off(tmp_path, ulps):
    """The device's reciprocal is an approximation within one ulp of 2^-24."""
    with open(os.path.join(ROOT, "sw2_gb300", "csrc", "sigmath.cuh")) as f:
        text = f.read()
    exact = "return 1.0f / f;"
    assert text.count(exact) == 1
    (tmp_path / "sigmath.cuh").write_text(text.replace(exact, f"return 1.0f / f + ({ulps}) * 0x1p-24f;"))
    assert host_run(tmp_path, DIV, 20_000_000) == ["0"]


CHECK = r"""
int main(int, char** argv) {  // the self-check's draws
  long long n = 0, far = 0;
  for (long long i = 0; i < atoll(argv[1]); i++) {
    const double b = from(((uint64_t)(1003 + next() % 80) << 52) | frac());
    double a;
    if (next() % 2) a = from(((uint64_t)(73 + next() % 1010) << 52) | frac());
    else a = b * (from(((uint64_t)(523 + next() % 500) << 52) | frac()) * (1 + std::ldexp((double)(next() % 8 + 1), -54)));
    if (next() % 64 == 0) a = from(((uint64_t)(900 + next() % 100) << 52) | (frac() >> 26 << 26));  // products that end in a tie
    n += sig_mismatches(a, i % 64 ? b : from(0x3ff0000000000000ULL | 1ULL << 51), sig_recip(bits(i % 64 ? b : 1.5)));
  }
  for (uint32_t u = 0; u < (1u << 23); u++) {
    SigFloat f;
    f.u = 0x3f800001u + u;
    far += !sig_rcp_close(f.f);
  }
  printf("%d %d\n", n != 0, far != 0);
}
"""


@GXX
@pytest.mark.parametrize("right,wrong,told", [
    ("", "", ["0", "0"]),
    ("0x20000u - 700u", "0x20000u", ["1", "0"]),        # sig_div: digits that came out low
    ("mid >= 0xff800000u", "false", ["1", "0"]),        # sig_div_known: an estimate that came out low
    ("m &= ~1ULL;", ";", ["1", "0"]),                   # sig_mul: ties
    ("- SIG_BIAS + ((sh", "- SIG_BIAS + (1u << 20) + ((sh", ["1", "0"]),
    ("return 1.0f / f;", "return 1.0f / f - 3 * 0x1p-24f;", ["1", "1"]),
])
def test_self_check_tells_planted_mistakes(tmp_path, right, wrong, told):
    """sw2g_selfcheck_division's comparison, with mistakes planted in a host copy."""
    with open(os.path.join(ROOT, "sw2_gb300", "csrc", "sigmath.cuh")) as f:
        text = f.read()
    if right:
        assert text.count(right) == 1
        text = text.replace(right, wrong)
    (tmp_path / "sigmath.cuh").write_text(text)
    assert host_run(tmp_path, CHECK, 4_000_000) == told


@pytest.mark.gpu
def test_gpu_quotients_and_products_match_ieee():
    """Divisors whose leading 24 bits round up to 2 or to the least above 1, and
    those of every exponent the metric factors may have."""
    rng = np.random.default_rng(17)
    low = rng.integers(0, 1 << 29, 4000, dtype=np.uint64)
    ones = np.uint64(0x3FF0000000000000) | np.uint64(((1 << 23) - 1) << 29) | low
    none = np.uint64(0x3FF0000000000000) | low
    d = np.concatenate([ones.view(np.float64), none.view(np.float64),
                        np.ldexp(rng.uniform(1.0, 2.0, 8000), rng.integers(-20, 60, 8000))])
    assert lib.selfcheck_division(d, samples=20_000, seed=14) == 0


def same_steps(case, counts, flags=0, raw=False):
    s = lib.Solver(case.params, flags=flags)
    s.upload(*case.fields(), mode=lib.UPLOAD_RAW if raw else lib.UPLOAD_FRAME)
    o = orc.Oracle(case.params, lape_eta=bool(flags & lib.FLAG_LAPE_ETA))
    o.load(case.fields(), raw=raw)
    for n in counts:
        assert s.step(n) == lib.OK
        assert o.step(n) == (0, -1)
        got = s.download()
        for k in ("eta", "u", "v", "tracer"):
            assert bitwise(got[k], o.field(k)), (k, s.steps_done())
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("sch", [1, 9])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_gpu_courant_number_of_one_matches_oracle(sch, sign):
    """v*Dt = DYN exactly in every row, so 1 - C is a zero, and fields that are
    zero beside steps of 64 and more: a face's slope term is a zero there."""
    case = cases.make_case(nx=64, ny=33, sch=sch, seed=3, jet="none", bumps=0, lat0=-30.0, lat1=20.0)
    p = case.params
    p.rP, p.depth, p.Dt, p.CFL = p.rE, 0.0, 512.0, 1e30
    g = cases.Grid(p)
    dyn = np.array([(g.lat1 - g.lat0) / p.ny * g.rM(g.latc(j)) for j in range(-1, p.ny + 3)])
    vj = sign * dyn / p.Dt
    assert np.all(np.abs(vj) * p.Dt / dyn == 1.0)
    case.v[:] = vj[:, None]
    case.eta[:] = 0.0
    for k, x in enumerate((case.eta, case.u, case.tracer)):
        x[12:20, 10:30] = (1000.0, 64.0, 3e5)[k]
        x[24, 5:50] = -128.0
    for x in (case.eta, case.u, case.v, case.tracer):
        cases.halo_wrap(x)
    same_steps(case, (1,), raw=True)


@pytest.mark.gpu
@pytest.mark.parametrize("tau", [1e20, 1e6])
@pytest.mark.parametrize("sch", [0, 2, 9])
def test_gpu_zero_sums_of_a_diverging_flow_are_plus_zero(sch, tau):
    """A layer of thickness zero in a flow away from a point: each cell's four
    terms are zeros, of signs such that a sum without the unused sides' zeros is
    -0; the reference's, which starts from +0, is +0. Only the histories of a
    checkpoint show it: eta + (-0) = eta."""
    case = cases.make_case(nx=64, ny=33, sch=sch, seed=3, jet="none", bumps=0, lat0=-30.0, lat1=20.0, hyper=False, Tau=tau)
    p = case.params
    p.depth, p.CFL = 0.0, 1e30
    case.eta[:] = 0.0
    case.u[:] = (np.arange(p.nx + 4) - 30.5)[None, :]
    case.v[:] = (np.arange(p.ny + 4) - 15.5)[:, None]
    for x in (case.u, case.v):
        cases.halo_wrap(x)
    s = lib.Solver(p)
    s.upload(*case.fields(), mode=lib.UPLOAD_RAW)
    assert s.step(1) == lib.OK
    S = (p.nx + 4) * (p.ny + 4)
    history = s.checkpoint()[-8 * S:][:S].reshape(p.ny + 4, p.nx + 4)  # of eta's tendency, the step's
    assert not np.any(history) and not np.any(np.signbit(history))


def rough_case(nx, ny, lat, orders=(1, 1, 1), **kw):
    """Rough velocities everywhere, wall rows included, and a tracer."""
    rng = np.random.default_rng(nx + ny)
    case = cases.make_case(nx=nx, ny=ny, sch=2, seed=3, jet="none", bumps=0, lat0=-lat, lat1=lat, tracer=True, cfl=0.05, **kw)
    nu4 = case.params.hypernu[1]
    case.params.hypernu = (orders[0] * 0.02 * nu4 ** 0.5, orders[1] * nu4, orders[2] * 0.05 * nu4 ** 1.5)
    case.params.CFL = 1e30
    for x in (case.u, case.v):
        x[:] = 0.1 * rng.standard_normal(x.shape)
        cases.halo_wrap(x)
    return case


def launches_of_a_step(case):
    s = lib.Solver(case.params)
    s.upload(*case.fields(), mode=lib.UPLOAD_RAW)
    assert s.step(2) == lib.OK and s.step(1) == lib.OK
    return s.last_launches()


@pytest.mark.gpu
@pytest.mark.parametrize("lat,nx,ny,wall", [(89.8, 64, 33, 0.0), (89.0, 33, 89, 1.0), (70.0, 40, 5, 1.0), (80.0, 31, 7, 0.0)])
def test_gpu_bands_next_to_a_pole_keep_the_merged_launch(lat, nx, ny, wall):
    """The row above the wall lies beyond the pole, where the metric factor of y
    turns negative and that of DYN(ny) + DYN(ny+1) is next to zero: only the wall
    row of v divides by it."""
    case = rough_case(nx, ny, lat)
    assert case.params.lat1 + 1.5 * (2 * lat) / ny > 90.0
    case.v[ny + 1] *= wall
    same_steps(case, (1, 1, 1), raw=True)
    assert launches_of_a_step(case) == launches_of_a_step(rough_case(nx, ny, 40.0))


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [1e-45, 1e-300])
def test_gpu_coefficients_outside_the_integer_range_keep_the_merged_launch(nu):
    """A hyperviscosity coefficient that the integer-pipe products do not take
    concerns that product alone."""
    case = rough_case(64, 33, 60.0, hyper=False)
    case.params.hypernu = (nu, 0.0, 0.0)
    same_steps(case, (1, 1, 1, 2), raw=True)
    assert launches_of_a_step(case) == launches_of_a_step(rough_case(64, 33, 60.0, orders=(1, 0, 0)))


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [4095, 4096, 4097, 8193])
@pytest.mark.parametrize("field", ["u", "v"])
def test_gpu_cfl_maximum_is_found_in_every_column(nx, field):
    """A warp takes 4096 columns of the CFL maxima: the one fast cell of the
    grid at their edges."""
    for col in sorted({1, min(nx, 4096), min(nx, 4097), nx}):
        case = cases.make_case(nx=nx, ny=6, sch=2, seed=3, jet="none", bumps=0, lat0=-30.0, lat1=20.0, hyper=False)
        p = case.params
        for x in (case.eta, case.u, case.v):
            x[:] = 0.0
        x = getattr(case, field)
        x[4, col + 1] = 1e-3
        cases.halo_wrap(x)
        g = cases.Grid(p)
        lat = g.latc(3)
        d = (g.lon1 - g.lon0) / nx * g.rZ(lat) if field == "u" else (g.lat1 - g.lat0) / p.ny * g.rM(lat)
        for slack, want in ((1.0001, lib.OK), (0.9999, lib.ERR_CFL)):
            p.CFL = p.Dt * 1e-3 / d * slack
            s = lib.Solver(p)
            s.upload(*case.fields(), mode=lib.UPLOAD_RAW)
            assert s.step(1) == want, (col, slack)


@pytest.mark.gpu
def test_gpu_wide_grid_takes_no_longer_than_a_square_one():
    """As many cells in 16 rows: no kernel's strips grow with the row."""
    ms = []
    for nx, ny in ((1024, 1024), (65536, 16)):
        case = cases.make_case(nx, ny, sch=2, seed=3, bumps=1, cfl=0.2)
        s = lib.Solver(case.params)
        s.upload(*case.fields())
        assert s.step(3) == lib.OK
        t = []
        for _ in range(7):
            assert s.step(5) == lib.OK
            t.append(s.last_step_ms())
        ms.append(min(t))
    assert ms[1] < 1.5 * ms[0]


@pytest.mark.gpu
@pytest.mark.parametrize("change", [dict(hypernu=(np.inf, 0.0, 0.0)), dict(hypernu=(0.0, np.nan, 0.0)), dict(hypernu=(0.0, 0.0, np.inf)),
                                    dict(gE=np.inf), dict(gE=np.nan)])
def test_gpu_constants_that_are_not_finite_fail_as_in_the_oracle(change):
    """A layer at rest: a zero times infinity or NaN is NaN, and the step's check finds it."""
    case = cases.make_case(nx=40, ny=24, sch=2, seed=3, jet="none", bumps=0, hyper=False)
    for x in (case.eta, case.u, case.v):
        x[:] = 0.0
    p = case.params
    p.CFL = 1e30
    for k, v in change.items():
        setattr(p, k, v)
    s = lib.Solver(p)
    s.upload(*case.fields(), mode=lib.UPLOAD_RAW)
    o = orc.Oracle(p)
    o.load(case.fields(), raw=True)
    rc, _ = o.step(1)
    assert s.step(1) == {1: lib.ERR_CFL, 2: lib.ERR_NONFINITE}[rc]


@pytest.mark.gpu
@pytest.mark.parametrize("sch", [5, 6])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("side", [1, -1])
def test_gpu_skipped_sides_that_are_not_finite_match_oracle(sch, axis, side):
    """No velocity anywhere, and a difference so small beside its neighbour that
    the square of the limiter's ratio overflows: zero times NaN is NaN."""
    case = cases.make_case(nx=64, ny=33, sch=sch, seed=3, jet="none", bumps=0, hyper=False)
    for x in (case.eta, case.u, case.v):
        x[:] = 0.0
    t = np.zeros(12)
    t[3], t[5] = 1.0, 1e-200  # ratios of 1/1e-200 on one side of the face between cells 4 and 5
    if side < 0:
        t = t[::-1]
    if axis:
        case.tracer[15, 20:32] = t
    else:
        case.tracer[10:22, 25] = t
    case.tracer[5, 50] = 1.0
    cases.halo_wrap(case.tracer)
    s = same_steps(case, (1,), raw=True)
    assert np.any(np.isnan(s.download()["tracer"]))
