"""fhd_flux_stag from the second call of a context on: the stress and face kernels over the
context's scratch, which calls on any stream take in turn."""
import ctypes
import time

import pytest
import torch

from fhdex_b200.context import Context
from fhdex_b200.params import argon, stable_dt
from fhdex_b200.state import StagState, StepNoise

pytestmark = pytest.mark.gpu


def prepared(p, steps=2):
    """A state some steps into a run, with its coefficients, and a noise W."""
    st = StagState(p, "cuda")
    ctx = Context(p)
    ctx.init_state(st)
    for s in range(steps):
        ctx.rk3_step(st, stable_dt(p), s)
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
