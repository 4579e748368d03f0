"""Products and quotients on the integer pipe (sigmath.cuh) and the FP64 step
where its kernels leave their usual path: values far outside the range of the
integer-pipe operations, sums that are zero, a flow that starts at rest, small
and ragged grids. The step is compared with the CPU oracle bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import oracle as orc
from sw2_gb300 import cases, lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "sigmath.cuh"
using namespace sw2g;
static uint64_t st = 0xA4093822299F31D0ULL;
static uint64_t next() {  // SplitMix64
  uint64_t z = (st += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
static double from(uint64_t b) { double d; std::memcpy(&d, &b, 8); return d; }
static uint64_t bits(double d) { uint64_t b; std::memcpy(&b, &d, 8); return b; }
static uint64_t frac() {  // random significands and the structured ones that make ties and carries
  const uint64_t F = (1ULL << 52) - 1, r = next();
  switch (next() % 8) {
    case 0: return r & 15;
    case 1: return F - (r & 15);
    case 2: return r & F & ~((1ULL << (r >> 59)) - 1);
    case 3: return (r & F) >> 26 << 26;
    case 4: return (r & F) >> 40 << 40;
    default: return r & F;
  }
}
int main(int argc, char** argv) {
  const long long n = atoll(argv[1]);
  long long bad[4] = {0, 0, 0, 0};
  for (long long i = 0; i < n; i++) {
    uint64_t A = ((uint64_t)(520 + next() % 1000) << 52) | frac(), B = ((uint64_t)(520 + next() % 1000) << 52) | frac();
    const int k = next() % 8;
    if (k < 2) A = bits(from(B) * from(0x3ff0000000000000ULL | frac()));  // quotients with few digits
    if (k == 2)  // quotients next to a rounding midpoint
      A = bits(from(B) * (from(0x3ff0000000000000ULL | frac()) + std::ldexp((double)(next() % 8 + 1), -54)));
    if (k == 3) A = B + next() % 7 - 3;
    const double a = from(A), b = from(B);
    if (std::isnormal(a * b) && std::isnormal(a * b * 0.5)) {
      bad[0] += sig_mul(A, B) != bits(a * b);
      bad[1] += sig_mul(A, B, 0xfff00000u) != bits(a * b * 0.5);
    }
    if (std::isnormal(a / b)) {
      bad[2] += sig_div(A, B) != bits(a / b);
      bad[3] += sig_div_known(A, B, sig_recip(B)) != bits(a / b);
    }
  }
  // significands within 600 ulps of 1 and 2 on both sides: the longest carries
  for (int i = 0; i < 1200; i++)
    for (int j = 0; j < 1200; j++) {
      const uint64_t A = 0x4000000000000000ULL - 600 + i, B = 0x4000000000000000ULL - 600 + j;
      bad[0] += sig_mul(A, B) != bits(from(A) * from(B));
      bad[2] += sig_div(A, B) != bits(from(A) / from(B));
      bad[3] += sig_div_known(A, B, sig_recip(B)) != bits(from(A) / from(B));
    }
  printf("%lld %lld %lld %lld\n", bad[0], bad[1], bad[2], bad[3]);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_products_and_quotients_match_ieee_on_the_host(tmp_path):
    c = tmp_path / "sig.cpp"
    c.write_text(HARNESS)
    exe = tmp_path / "sig"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-I",
                    os.path.join(ROOT, "sw2_gb300", "csrc"), "-o", str(exe), str(c)], check=True)
    out = subprocess.run([str(exe), str(20_000_000)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0"] * 4


def bitwise(a, b):
    """Equal bit for bit, NaNs as NaNs."""
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan]) and np.array_equal(np.isnan(a), np.isnan(b))


def same_steps(case, counts, flags=0, fields=("eta", "u", "v", "tracer")):
    s = lib.Solver(case.params, flags=flags)
    s.upload(*case.fields(), mode=lib.UPLOAD_FRAME)
    o = orc.Oracle(case.params)
    o.load(case.fields())
    for n in counts:
        assert s.step(n) == lib.OK
        assert o.step(n) == (0, -1)
        got = s.download()
        for k in fields:
            assert bitwise(got[k], o.field(k)), (k, s.steps_done())


@pytest.mark.gpu
@pytest.mark.parametrize("sch", [0, 1, 2, 4, 5, 6, 7, 8, 9])
def test_gpu_flow_from_rest_matches_oracle(sch):
    """A bump with a sharp edge in a layer at rest: exact zeros ahead of the
    front, and behind it values from normal down through the subnormals."""
    case = cases.make_case(nx=150, ny=70, sch=sch, seed=4, jet="none", bumps=0, tracer=False)
    case.eta[30:40, 40:60] += 50.0
    case.tracer[32:36, 44:50] = 0.5
    cases.halo_wrap(case.eta)
    cases.halo_wrap(case.tracer)
    # limiters 5 and 6 square the slope ratio, which overflows (a NaN, and an
    # abort, in the reference as well) once the tails are tiny
    same_steps(case, (1, 1, 1, 5, 20, 30) if sch not in (5, 6) else (1, 1, 1, 5))


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-40, 1e-100, 1e-160, 1e-270, 1e-305])
def test_gpu_tiny_velocities_match_oracle(scale):
    """Velocities whose differences, products and Courant numbers lie below
    the exponents the integer-pipe operations take, next to ordinary ones."""
    rng = np.random.default_rng(11)
    case = cases.make_case(nx=97, ny=40, sch=1, seed=6, jet="none", bumps=0, tracer=True, TracerDis=1e-6)
    case.eta[:] = 0.0
    case.u[:] = scale * rng.standard_normal(case.u.shape)
    case.v[:] = scale * rng.standard_normal(case.v.shape)
    case.u[10:14, 20:60] = 3.0
    case.tracer[20:24, 30:50] = scale
    for x in (case.u, case.v, case.tracer):
        cases.halo_wrap(x)
    same_steps(case, (1, 1, 1, 2))


@pytest.mark.gpu
def test_gpu_mixed_magnitudes_match_oracle():
    """Cells of every magnitude side by side: 2^-1000 .. 2^20, and zeros of both signs."""
    rng = np.random.default_rng(3)
    case = cases.make_case(nx=130, ny=48, sch=2, seed=9, jet="none", bumps=1, tracer=True)
    for x in (case.u, case.v):
        x[:] = np.ldexp(rng.standard_normal(x.shape), rng.integers(-1000, 5, x.shape))
        x[rng.random(x.shape) < 0.2] = 0.0
        x[rng.random(x.shape) < 0.1] = -0.0
        cases.halo_wrap(x)
    same_steps(case, (1, 1, 1, 1))


@pytest.mark.gpu
def test_gpu_metrics_outside_the_integer_range_match_oracle():
    """A planet so small that the metric factors fall below the divisors the
    integer-pipe quotients take: the literal kernels and the FP64 unit."""
    case = cases.make_case(nx=40, ny=24, sch=2, seed=2, jet="none", bumps=0)
    p = case.params
    p.rE = p.rP = 1e-7
    p.Dt, p.CFL, p.hypernu = 1e-12, 1e30, (0.0, 0.0, 0.0)
    case.eta[8:12, 10:20] += 1e-3
    cases.halo_wrap(case.eta)
    same_steps(case, (1, 1, 2))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(3, 3), (4, 4), (5, 3), (30, 8), (31, 9), (32, 33), (61, 5), (62, 17), (124, 3), (125, 40)])
@pytest.mark.parametrize("orders", [(0, 1, 0), (1, 0, 0), (1, 1, 1), (0, 0, 1)])
def test_gpu_laplacians_on_edge_sizes_match_oracle(nx, ny, orders):
    """The marching Laplacian kernels at the edges of their strips (30 and 31
    columns, 1 to 8 rows), one to three levels, the last one inside the eta
    kernel; halos included."""
    wind = np.stack([np.arange(-180.0, 181.0), 5 * np.cos(np.deg2rad(np.arange(-180.0, 181.0)))], axis=1)
    case = cases.make_case(nx=nx, ny=ny, sch=2, seed=nx + ny, bumps=1, sigma_km=(20000.0, 20000.0), cfl=0.05,
                           wind=wind if nx == 62 else None)
    nu4 = case.params.hypernu[1]
    case.params.hypernu = (orders[0] * 0.02 * nu4 ** 0.5, orders[1] * nu4, orders[2] * 0.05 * nu4 ** 1.5)
    same_steps(case, (1, 1, 1, 3))
