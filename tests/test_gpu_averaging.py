"""Driving-force averaging ($Average Yes, the reference default) on the GPU.

The oracle's restatement of DrivingForce::Average is pinned to the reference by the fixtures
tests/golden/average_*.npz (tests/test_oracle.py); here the CUDA path (opgpu_set_averaging) is held
to the oracle and to those fixtures.  The device decides per pair and voxel whether the averaged force
is the raw force or none, and takes the pair's tabulated force; the reference's quotient of sums
differs from it by rounding: the bar is the parity bar (identical lists, borderline voxels counted,
max|dphi| <= 1e-9) over the tested windows.
"""
from pathlib import Path

import numpy as np
import pytest

from openphase_b200.cases import Case
from openphase_b200.context import Context
from oracle.bridge import Oracle, positive_entries
from tests.golden.make_golden import GOLDEN_CASES
from tests.parity import compare_states

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"
TOL = 1e-9


@pytest.mark.parametrize("name", ["average_20", "average_eta6_24"])
def test_averaging_matches_reference_fixture_and_oracle(name):
    case, steps = GOLDEN_CASES[name]
    z = np.load(GOLDEN / f"{name}.npz")
    state = case.initial_state()
    ctx = Context.from_case(case, precision="fp64", k_slots=16, state=state)
    ora = Oracle(case, *state)
    prev = 0
    for s in steps:
        st = ctx.step(case.dt, s - prev)
        ora.step(s - prev)
        prev = s
        assert st & 0b11 == 0 and not st & (1 << 7), st
        gpu = ctx.download()
        ref = positive_entries(z[f"s{s}_counts"].astype(np.int32), z[f"s{s}_idx"].astype(np.int32), z[f"s{s}_val"])
        for other in (ref, ora.state(positive_only=True)):
            r = compare_states(gpu, other, case.ngrains)
            assert r["non_borderline_mismatch_voxels"] == 0 and r["max_dphi"] <= TOL, (s, r)


def test_averaging_larger_grid():
    case = Case(48, 40, 32, 14, seed=31, iwidth=5.0, dt=0.08, sigma=1.2, sigma_pairs=(0.8, 0.4), dg_scale=0.15,
                average=True, name="average_48")
    state = case.initial_state()
    tiled = Context.from_case(case, precision="fp64", k_slots=16, state=state)
    ora = Oracle(case, *state)
    plain = Context.from_case(case.with_(average=False), precision="fp64", k_slots=16, state=state)
    prev = 0
    for s in (1, 10, 30):
        tiled.step(case.dt, s - prev)
        plain.step(case.dt, s - prev)
        ora.step(s - prev)
        prev = s
        r = compare_states(tiled.download(), ora.state(positive_only=True), case.ngrains)
        assert r["non_borderline_mismatch_voxels"] == 0 and r["max_dphi"] <= TOL, (s, r)
    # averaging is not a rounding-level change: pairs far from their interface core lose their force
    r = compare_states(tiled.download(), plain.download(), case.ngrains)
    assert r["max_dphi"] > 1e-3, r


def test_averaging_refused_where_unsupported():
    from openphase_b200._lib import E_INVALID, OpgpuError
    from openphase_b200.adjoint import Rollout
    case, _ = GOLDEN_CASES["average_20"]
    ctx = Context.from_case(case, precision="fp64", k_slots=16)
    R = Rollout(ctx, case.dt, 4)
    R.forward()
    with pytest.raises(OpgpuError) as e:
        R.backward(np.ones(case.ngrains))
    assert e.value.code & E_INVALID


# junction-dense small grains (up to 13 fields a voxel: every word of the pair mask; VolumeRatio < 1
# lowers the threshold, so voxels hold several pairs above it), and boxes the sphere wraps around
DENSE = {
    "dense": Case(24, 24, 24, 30, seed=7, iwidth=6.0, dt=0.08, sigma=1.2, sigma_pairs=(0.8, 0.4), dg_scale=0.05,
                  average=True, name="dense"),
    "thin_box": Case(26, 11, 5, 6, seed=13, iwidth=6.0, dt=0.08, dg_scale=0.1, average=True, name="thin_box"),
    "narrow": Case(24, 20, 22, 9, seed=17, iwidth=4.0, dt=0.08, dg_scale=0.1, average=True, name="narrow"),
}


@pytest.mark.parametrize("name", list(DENSE))
@pytest.mark.parametrize("variant", ["tiled", "generic"])
def test_averaging_dense_and_wrapped_grids(name, variant):
    case = DENSE[name]
    state = case.initial_state()
    ctx = Context.from_case(case, precision="fp64", k_slots=16, state=state)
    ctx.set_kernel_variant(variant)
    ora = Oracle(case, *state)
    for _ in range(4):
        ctx.step(case.dt, 1)
        ora.step(1)
        r = compare_states(ctx.download(), ora.state(positive_only=True), case.ngrains)
        assert r["non_borderline_mismatch_voxels"] == 0 and r["max_dphi"] <= TOL, r


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("threshold", [0.0, 0.02])
def test_averaging_tiled_equals_generic(precision, threshold):
    """Both kernels read the same mask: large grains (VolumeRatio = 1) give identical lists and values
    bit for bit; a low threshold makes most marks "several"."""
    case = Case(40, 33, 37, 10, seed=19, iwidth=5.0, dt=0.08, dg_scale=0.1, average=True, name="tiled_generic")
    state = case.initial_state()
    got = []
    for variant in ("tiled", "generic"):
        ctx = Context.from_case(case, precision=precision, k_slots=12, state=state)
        ctx.set_averaging(True, 0, threshold)
        ctx.set_kernel_variant(variant)
        ctx.step(case.dt, 3)
        got.append(ctx.download())
    r = compare_states(*got, case.ngrains)
    assert r["same_sets"] and r["max_dphi"] == 0.0, r


def _marks(case, state, threshold):
    """Per voxel the pair above the threshold (VolumeRatio = 1) as a key, and whether it has several."""
    counts, idx, val = state
    starts = np.concatenate([[0], np.cumsum(counts)])
    key, several = np.zeros(case.n, np.int64), np.zeros(case.n, bool)
    bar = np.sqrt(threshold * (1.0 - threshold))
    for u in np.nonzero(counts > 1)[0]:
        g, x = idx[starts[u]:starts[u + 1]], val[starts[u]:starts[u + 1]]
        a, b = np.nonzero(np.triu(np.sqrt(np.outer(x, x)) > bar, 1))
        if a.size:
            key[u] = 1 + min(g[a[0]], g[b[0]]) * case.ngrains + max(g[a[0]], g[b[0]])
            several[u] = a.size > 1
    return key, several


# One case for each way a mask is found: (case, range, threshold, what the first state has to show).
# A tile of 8 x 8 x 16 voxels takes 4608 marks of 256 grain pairs from its halo, no voxel with several
# pairs above the threshold, and a radius of 16; whatever is beyond that is searched voxel by voxel.
_BOX = dict(dt=0.08, sigma=1.2, dg_scale=0.1, average=True)
ROUTES = {
    "range_17": (Case(20, 18, 22, 6, seed=23, iwidth=5.0, name="range_17", **_BOX), 17, 0.0, None),
    "range_12": (Case(24, 22, 26, 8, seed=29, iwidth=5.0, name="range_12", **_BOX), 12, 0.0, None),
    "many_marks": (Case(24, 24, 24, 30, seed=7, iwidth=6.0, name="many_marks", **_BOX), 8, 0.0,
                   lambda m, k, s: m > 4608 and k <= 256 and not s),
    "many_pairs": (Case(32, 32, 32, 150, seed=7, iwidth=4.0, name="many_pairs", **_BOX), 7, 0.45,
                   lambda m, k, s: m <= 4608 and k > 256 and not s),
    "several": (Case(24, 20, 22, 9, seed=17, iwidth=5.0, name="several", **_BOX), 0, 0.02, lambda m, k, s: s),
}


@pytest.mark.parametrize("name", list(ROUTES))
def test_averaging_every_route_matches_oracle(name):
    """Ranges, thresholds and grain sizes that send the search through each of its routes, with a nucleus
    volume so small that every VolumeRatio is 1: the volumes' summation order plays no part."""
    case, reach, threshold, expected = ROUTES[name]
    state = case.initial_state()
    factor = 0.01
    ora = Oracle(case, *state, nucleus_volume_factor=factor, average_range=reach, average_threshold=threshold)
    assert (ora.grains()["volume_ratio"] == 1.0).all()
    if expected:
        r = reach or int(case.iwidth)
        shape = (case.nx, case.ny, case.nz)
        key, several = _marks(case, ora.state(positive_only=True), threshold or 1.0 / 3.0)
        at = np.ix_(*(np.arange(-r, t + r) % n for t, n in zip((8, 8, 16), shape)))
        halo = key.reshape(shape)[at]
        assert expected((halo > 0).sum(), np.unique(halo[halo > 0]).size, several.reshape(shape)[at].any())
    ctx = Context(case.nx, case.ny, case.nz, iwidth=case.iwidth, stencil=case.stencil, precision="fp64", k_slots=16)
    ctx.set_model(case.sigma_phase(), case.mu_phase(), limit=case.limit_phase(), nucleus_volume_factor=factor)
    ctx.set_grains(case.ngrains)
    ctx.set_driving_force(case.driving_force())
    ctx.set_averaging(True, reach, threshold)
    ctx.upload(*state)
    ctx.finalize_initialization()
    for _ in range(3):
        assert ctx.step(case.dt, 1) & 0b11 == 0
        ora.step(1)
        r = compare_states(ctx.download(), ora.state(positive_only=True), case.ngrains)
        assert r["non_borderline_mismatch_voxels"] == 0 and r["max_dphi"] <= TOL, r
