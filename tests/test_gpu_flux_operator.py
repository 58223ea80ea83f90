"""fhd_flux_stag from the second call of a context on: the stress and face kernels over the
context's scratch, which calls on any stream take in turn."""
import ctypes
import time

import pytest
import torch

from fhdex_b200.context import Context
from fhdex_b200.params import argon, argon_single, mixture4, stable_dt, with_walls
from fhdex_b200.state import StagState, StepNoise
from tests.helpers import compare_named
from tests.test_gpu_lowdim import CASES as LOWDIM, DT as LOWDIM_DT
from tests.test_gpu_walls import CASES as WALLS, DT as WALLS_DT

pytestmark = pytest.mark.gpu

CASES = {
    "argon": lambda: argon((9, 8, 7), dx=8e-6, seed=81),
    "argon_adv0_visc3": lambda: argon((8, 9, 7), dx=8e-6, advection_type=0, visc_type=3, zeta_ratio=0.5, seed=82),
    "argon_adv1": lambda: argon((7, 9, 8), dx=8e-6, advection_type=1, seed=83),
    "argon_no_noise": lambda: argon((9, 8, 7), dx=8e-6, stoch_stress_form=0, seed=84),
    "single": lambda: argon_single((6, 7, 9), dx=8e-6, seed=85),
    "mixture4": lambda: mixture4((7, 6, 5), dx=8e-6, seed=86),
    "mixture4_large": lambda: mixture4((41, 37, 33), dx=8e-6, seed=87),
    **WALLS,
    **LOWDIM,
}
# more faces than the SMs hold threads at once: the face kernel's grid of these runs
LARGE = {
    "large_1d": lambda: argon((250, 33, 32), dx=8e-6, seed=91).replace(do_1D=1),
    "large_2d_walls": lambda: with_walls(mixture4((129, 130, 16), dx=8e-6, seed=92),
                                         x=dict(vel=2, therm=2, mass=1, t=(263.0, 283.0))).replace(do_2D=1),
}
CASES.update(LARGE)
DT = {**WALLS_DT, **LOWDIM_DT}


def prepared(p, steps=2, dt=None):
    """A state some steps into a run, with its coefficients, and a noise W."""
    st = StagState(p, "cuda")
    ctx = Context(p)
    ctx.init_state(st)
    for s in range(steps):
        ctx.rk3_step(st, dt or stable_dt(p), s)
    nz = StepNoise(p, "cuda")
    ctx.fill_step_noise(nz, steps)
    torch.cuda.synchronize()
    ctx.close()
    return st, nz


def operator(ctx, st, nz):
    ctx.flux_stag(st, nz.face[0], nz.edge[0], nz.cen[0], stable_dt(st.p))


def fluxes(st):
    return {n: m.arr for n, m in st.named(aux=True).items() if "flux" in n}


def poison(st):
    for a in fluxes(st).values():
        a.fill_(-7.0)


@pytest.mark.parametrize("name", list(CASES))
def test_later_calls_equal_the_first(name):
    """A context's first call computes in kernels of their own, which recompute every stress
    per face; the later ones go through the stage's kernels.  Bit for bit, on every box."""
    st, nz = prepared(CASES[name](), dt=DT.get(name))
    ctx = Context(st.p)
    operator(ctx, st, nz)
    first = {n: a.clone() for n, a in fluxes(st).items()}
    for _ in range(2):
        poison(st)
        operator(ctx, st, nz)
        for n, a in fluxes(st).items():
            assert torch.equal(a, first[n]), n
    assert ctx.status() == 0
    assert all(torch.isfinite(a).all() for a in first.values())
    ctx.close()


@pytest.mark.parametrize("injected", [False, True])
@pytest.mark.parametrize("name", list(WALLS) + list(LOWDIM) + list(LARGE))
def test_by_products_leave_the_step_as_without(name, injected):
    """Boxes with walls and quasi-1-D / 2-D runs: a step that returns its coefficients and
    fluxes leaves the state of one that does not, bit for bit."""
    st, nz = prepared(CASES[name](), dt=DT.get(name))
    out = []
    for aux in (False, True):
        d = st.clone()
        ctx = Context(st.p)
        for s in (2, 3):
            ctx.fill_step_noise(nz, s)
            ctx.rk3_step(d, DT.get(name) or stable_dt(st.p), s, noise=nz if injected else None, aux=aux)
        assert ctx.status() == 0
        ctx.close()
        out.append(d)
    bad, _ = compare_named(out[1].named(), out[0].named())
    assert not bad, bad[:6]


def test_calls_on_two_streams():
    """Calls that share the scratch from two streams in turn, each behind the other."""
    p = argon((44, 40, 36), dx=8e-6, seed=88)
    a, nz = prepared(p)
    b, _ = prepared(p.replace(seed=89), steps=3)
    ctx = Context(p)
    want = []
    for st in (a, b):
        fresh = Context(p)
        operator(fresh, st, nz)
        want.append({n: v.clone() for n, v in fluxes(st).items()})
        fresh.close()
        operator(ctx, st, nz)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    for _ in range(20):
        for s, st in zip(streams, (a, b)):
            with torch.cuda.stream(s):
                poison(st)
                operator(ctx, st, nz)
    torch.cuda.synchronize()
    for st, w in zip((a, b), want):
        for n, v in fluxes(st).items():
            assert torch.equal(v, w[n]), n
    assert ctx.status() == 0
    ctx.close()


def test_a_call_waits_for_the_last_on_a_recycled_stream():
    """A stream destroyed with the operator still running on it, and another one, which the
    driver may give the same handle: the second call takes the scratch after the first."""
    p = argon((24, 20, 16), dx=8e-6, seed=71)
    a, nz = prepared(p)
    b, _ = prepared(p.replace(seed=72), steps=3)
    ctx = Context(p)
    want = []
    for st in (a, b):
        for _ in range(2):
            operator(ctx, st, nz)
        want.append({n: v.clone() for n, v in fluxes(st).items()})
        poison(st)
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so.12")
    handles = []
    for st in (a, b):
        h = ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(h), 1) == 0
        handles.append(h.value)
        s = torch.cuda.ExternalStream(h.value)
        with torch.cuda.stream(s):
            if st is a:
                torch.cuda._sleep(600_000_000)     # some 0.3 s
            operator(ctx, st, nz)
            done = torch.cuda.Event()
            done.record()
        assert rt.cudaStreamDestroy(h) == 0
    time.sleep(0.05)
    assert not done.query(), "the second call did not wait for the first"
    torch.cuda.synchronize()
    for st, w in zip((a, b), want):
        for n, v in fluxes(st).items():
            assert torch.equal(v, w[n]), n
    assert ctx.status() == 0      # (and the context is back on a stream that exists)
    ctx.close()


def test_close_ends_the_scratch_s_last_use():
    """The operator on one stream, a later call on another, and close(): the first stream is
    done when close returns, and the scratch is back in the device's memory pool."""
    p = argon((24, 20, 16), dx=8e-6, seed=73)
    st, nz = prepared(p)
    ctx = Context(p)
    operator(ctx, st, nz)
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so.12")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0

    def in_use():
        assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0     # cudaMemPoolAttrUsedMemCurrent
        return used.value

    before = in_use()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(600_000_000)
        operator(ctx, st, nz)
        done = torch.cuda.Event()
        done.record()
    assert ctx.status() == 0      # on the current stream, which the context then keeps
    ctx.close()
    assert done.query()
    torch.cuda.synchronize()
    assert in_use() < before
