"""opgpu_pack_plane / opgpu_unpack_plane: the one-kernel copy (planes whose parts start on 16 bytes, device
buffers of the context's GPU) and the general copy give the bytes the layout states, both ways, and
checkpoints restore a state exactly."""
import numpy as np
import pytest

from openphase_b200._lib import E_STATE, OpgpuError
from openphase_b200.adjoint import Rollout
from openphase_b200.cases import Case
from openphase_b200.context import Context

pytestmark = pytest.mark.gpu

# (ny, nz): parts on 16 bytes; an odd plane (the general copy)
SHAPES = [(20, 12), (17, 13)]


def _ctx(ny, nz, precision, k):
    case = Case(10, ny, nz, 6, seed=5, iwidth=4.0, dt=0.1, name="planes")
    ctx = Context.from_case(case, precision=precision, k_slots=k)
    ctx.step(case.dt, 3)
    return case, ctx


def _unpacked(buf, m, k, real):
    count = buf[:m]
    grain = buf[m:m + 2 * k * m].copy().view(np.int16).reshape(k, m)
    value = buf[m + 2 * k * m:].copy().view(real).reshape(k, m)
    return count, grain, value


@pytest.mark.parametrize("ny,nz", SHAPES)
@pytest.mark.parametrize("precision,k", [("fp64", 8), ("fp32", 12)])
@pytest.mark.parametrize("shift", [0, 8])   # a buffer that starts off 16 bytes takes the general copy
def test_planes_hold_the_state_and_restore_it(ny, nz, precision, k, shift):
    import torch
    case, ctx = _ctx(ny, nz, precision, k)
    m, real = ny * nz, np.float32 if precision == "fp32" else np.float64
    counts, idx, val = ctx.download()
    starts = np.concatenate([[0], np.cumsum(counts)])
    size = ctx.plane_bytes()
    planes = [torch.zeros(size + shift, dtype=torch.uint8, device="cuda") for _ in range(case.nx)]
    for x, b in enumerate(planes):
        ctx.pack_plane(x, b.data_ptr() + shift)
        c, g, v = _unpacked(b[shift:].cpu().numpy(), m, k, real)
        assert np.array_equal(c, counts[x * m:(x + 1) * m])
        for u in range(m):
            lo = starts[x * m + u]
            assert np.array_equal(g[:c[u], u], idx[lo:lo + c[u]])
            assert np.array_equal(v[:c[u], u].astype(np.float64), val[lo:lo + c[u]])
    ctx.step(case.dt, 2)
    for x, b in enumerate(planes):
        ctx.unpack_plane(x, b.data_ptr() + shift)
    for a, b in zip(ctx.download(), (counts, idx, val)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_checkpoint_restores_the_stored_fields(precision):
    case, ctx = _ctx(17, 13, precision, 16)
    ctx.checkpoint_reserve(1)
    before = ctx.download()
    ctx.checkpoint_save(0)
    ctx.step(case.dt, 4)
    assert not np.array_equal(ctx.download()[2], before[2])
    ctx.checkpoint_load(0)
    for a, b in zip(ctx.download(), before):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_slots_that_were_never_saved_are_refused(precision):
    """A reserved slot's memory holds whatever the device memory held before: its counts are not to be
    trusted.  Loading it and stepping back to it are refused, and the state stays as it was."""
    case, ctx = _ctx(17, 13, precision, 8)
    w = np.ones(case.ngrains)
    ctx.checkpoint_reserve(3)
    ctx.checkpoint_save(0)
    before = ctx.download()
    ctx.adjoint_begin(w)
    for call in (lambda: ctx.checkpoint_load(1), lambda: ctx.adjoint_step(2, case.dt)):
        with pytest.raises(OpgpuError) as e:
            call()
        assert e.value.code & E_STATE
    for a, b in zip(ctx.download(), before):
        assert np.array_equal(a, b)
    ctx.step_save_input(case.dt, 1)   # the ways to fill a slot
    ctx.checkpoint_load(1)
    for a, b in zip(ctx.download(), before):
        assert np.array_equal(a, b)
    R = Rollout(ctx, case.dt, 5)      # its segment slots are new
    with pytest.raises(OpgpuError) as e:
        R.backward(w)
    assert e.value.code & E_STATE
    R.forward()
    R.backward(w)
    assert R.adjoint_status == 0


@pytest.mark.parametrize("grains", [(6, 40), (40, 6)])
def test_slots_and_sweeps_follow_the_number_of_grains(grains):
    """Checkpoints and adjoint buffers of a context that takes another number of grains: the slots hold no
    state, and forward and backward give what a new context gives."""
    def rollout(ctx, case):
        G = case.ngrains
        ctx.set_pair_table(np.ones((G, G)), np.ones((G, G)))
        R = Rollout(ctx, case.dt, 6)
        volume = R.forward()
        grads = R.backward(np.arange(G) - 0.5 * G)
        dv = R.tangent(None, None, np.arange(G) * 0.1)
        return [volume, *grads, dv]

    first, second = (Case(22, 20, 18, G, seed=G, iwidth=4.0, dt=0.08, dg_scale=0.05, name="regrain") for G in grains)
    ctx = Context.from_case(first, precision="fp64", k_slots=16)
    rollout(ctx, first)
    ctx.set_grains(second.ngrains)
    ctx.set_driving_force(second.driving_force())
    ctx.upload(*second.initial_state())
    ctx.finalize_initialization()
    for call in (lambda: ctx.checkpoint_load(0), lambda: ctx.adjoint_step(1, second.dt), lambda: ctx.tlm_step(second.dt)):
        with pytest.raises(OpgpuError) as e:
            call()
        assert e.value.code & E_STATE
    got = rollout(ctx, second)
    expected = rollout(Context.from_case(second, precision="fp64", k_slots=16), second)
    for a, b in zip(got, expected):   # up to the order of the atomic sums
        assert np.allclose(a, b, rtol=1e-9, atol=1e-9 * np.abs(b).max())
