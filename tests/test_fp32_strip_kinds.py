"""Momentum, mass and tracer strips of the FP32 form's main launch.

A batch runs its strips 16 to 64 rows high, of all three kinds as soon as one
member has an active tracer; a member stepped alone picks its own strip height,
and its strips are of two kinds without a tracer. Every face is computed with
the same operations wherever a strip begins, so both end on the same bits. The
sizes put a strip's edge on, before and after the grid's: 128 columns, 16 rows.
"""
import numpy as np
import pytest

from sw2_gb300 import cases, lib

pytestmark = pytest.mark.gpu


def make(nx, ny, sch, seed, winds, tracer):
    lat = np.arange(-180.0, 181.0)
    wind = np.stack([lat, 25 * np.cos(np.deg2rad(lat) * 3)], axis=1) if winds else None
    return cases.make_case(nx=nx, ny=ny, sch=sch, seed=seed, wind=wind, tracer=tracer, TracerDis=2.0e-6 if tracer else 0.0,
                           sigma_km=(6000.0, 6000.0))


def solver(case):
    s = lib.Solver(case.params, precision=lib.FP32)
    s.upload(*case.fields())
    return s


@pytest.mark.parametrize("sch", [1, 2])
@pytest.mark.parametrize("winds", [False, True])
@pytest.mark.parametrize("rows", lib.Batch.TILE_ROWS)
def test_members_with_and_without_tracer_match_stepped_alone(rows, winds, sch):
    sizes = [(3, 3), (127, 15), (128, 16), (129, 17), (257, 65)]
    members = [make(nx, ny, sch, 30 + k, winds and k % 2 == 0, k in (1, 3, 4)) for k, (nx, ny) in enumerate(sizes)]
    inside = [solver(c) for c in members]
    b = lib.Batch(inside)
    b.set_schedule(rows, "rows")
    assert b.step(6) == lib.OK
    for c, s in zip(members, inside):
        alone = solver(c)
        assert alone.step(6) == lib.OK
        got, ref = s.download(), alone.download()
        for k in ref:
            assert np.array_equal(got[k], ref[k], equal_nan=True), (c.params.nx, c.params.ny, k)
        assert np.all(np.isfinite(got["eta"]))
