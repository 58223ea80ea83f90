"""The stage pipeline's routes by size: periodic ghosts stored by the update and the
conversion or filled by a launch of their own, and the staged or the plain stress
kernel.  FP64 bit for bit against the oracle (ghosts included) and, on boxes too large
for it, against the fused stage kernel, which shares neither; the mixed path's ghosts
bit for bit against their valid points."""
import pytest
import torch

from fhdex_b200.batch import Batch
from fhdex_b200.context import Context
from fhdex_b200.params import argon, argon_single, mixture4, stable_dt
from fhdex_b200.state import StagState, StepNoise
from tests.helpers import compare_named, perturbed_state

pytestmark = pytest.mark.gpu


def mixture3(n, **kw):
    """Ar/Ne/He: an odd number of flux components in the packed operands."""
    return mixture4(n, **kw).replace(nspecies=3, molmass=(39.95, 20.18, 4.00), diameter=(3.66e-8, 2.58e-8, 2.18e-8),
                                     dof=(3.0,) * 3, e0=(0.0,) * 3, hcv=(-1.0,) * 3, hcp=(-1.0,) * 3,
                                     rhobar=(0.5, 0.25, 0.25))


GASES = {"single": argon_single, "argon": argon, "mixture3": mixture3, "mixture4": mixture4}


# two ghosts: images need more than four cells in each direction (5 the smallest box of
# them, 4 and 3 the launch of their own)
@pytest.mark.parametrize("gas,n", [("argon", (5, 5, 5)), ("argon", (4, 6, 7)), ("argon", (9, 5, 33)),
                                   ("argon", (16, 3, 5)), ("mixture3", (5, 6, 9)), ("mixture4", (6, 4, 5))])
def test_small_boxes_equal_oracle_bitwise(oracle, gas, n):
    p = GASES[gas](n, dx=8e-6, seed=61)
    st = perturbed_state(oracle, p, seed=62)
    d = st.clone(device="cuda")
    dt = stable_dt(p)
    ctx = Context(p)
    nz = StepNoise(p, "cuda")
    for s in range(3):
        ctx.fill_step_noise(nz, s)
        ctx.rk3_step(d, dt, s, aux=(s == 2))
        nzc = nz.to("cpu")
        torch.cuda.synchronize()
        assert oracle.rk3_step(st, nzc, dt) == 0
    assert ctx.status() == 0
    bad, _ = compare_named(d.named(aux=True), st.named(aux=True))
    assert not bad, bad[:6]
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("gas,n,ngc", [("argon", (5, 7, 33), 2), ("mixture3", (8, 7, 9), 3), ("argon", (6, 8, 7), 3),
                                       ("mixture4", (12, 5, 4), 2), ("single", (5, 6, 7), 2)])
def test_ghosts_are_periodic_images(gas, n, ngc, precision):
    p = GASES[gas](n, dx=8e-6, seed=63, precision=precision).replace(ngc=ngc)
    st = StagState(p, "cuda", aux=False)
    ctx = Context(p)
    ctx.init_state(st)
    ctx.rk3_steps(st, stable_dt(p), 0, 3)
    torch.cuda.synchronize()
    for name, m in st.named().items():
        a = m.arr
        for dim in (-1, -2, -3):
            cells = n[-1 - dim]
            i = torch.arange(a.shape[dim], device="cuda") - ngc
            top = a.shape[dim] - 2 * ngc - 1            # last valid index (the node of the high side when nodal)
            w = torch.where(i < 0, i + cells, torch.where(i > top, i - cells, i)) + ngc
            assert torch.equal(a, a.index_select(a.dim() + dim, w)), (name, dim)
    ctx.close()


# the staged stress kernel takes up to five waves of its blocks, about 76^3 points: both
# sides of the line, ragged, and a box of one block's remainder
@pytest.mark.parametrize("n", [(71, 72, 73), (83, 84, 85), (9, 4, 3)])
@pytest.mark.parametrize("kw", [{}, dict(advection_type=0, visc_type=3, zeta_ratio=0.5), dict(stoch_stress_form=0)])
def test_stress_kernels_equal_fused_stage_bitwise(n, kw):
    p = argon(n, dx=8e-6, seed=64, **kw)
    dt = stable_dt(p)
    fused = next(t for t, name in enumerate(Context.tiles()) if name.startswith("fused"))
    out = []
    for t in (-1, fused):
        st = StagState(p, "cuda", aux=False)
        ctx = Context(p)
        if t >= 0:
            ctx.set_tile(t)
        ctx.init_state(st)
        ctx.rk3_steps(st, dt, 0, 2)
        assert ctx.status() == 0
        out.append(st)
        ctx.close()
    bad, _ = compare_named(out[0].named(), out[1].named())
    assert not bad, bad[:6]


@pytest.mark.parametrize("persistent", [False, True])
def test_batch_with_a_member_too_small_for_images(persistent):
    """One member of four cells across sends every member's ghosts to the ghost launch."""
    ps = [argon((12, 9, 10), dx=8e-6, seed=65), argon((4, 6, 8), dx=8e-6, seed=66)]
    dts = [stable_dt(p) for p in ps]
    b = Batch(2, 0)
    sts = [StagState(p, "cuda", aux=False) for p in ps]
    for p, st, dt in zip(ps, sts, dts):
        b.add(p, st, dt)
    b.set_persistent(persistent)
    b.step(2)
    torch.cuda.synchronize()
    for p, st, dt in zip(ps, sts, dts):
        r = StagState(p, "cuda", aux=False)
        ctx = Context(p)
        ctx.init_state(r)
        for s in range(2):
            ctx.rk3_step(r, dt, s, aux=False)
        torch.cuda.synchronize()
        bad, _ = compare_named(st.named(), r.named())
        assert not bad, bad[:6]
        ctx.close()


def test_flux_operator_under_capture_equals_eager():
    """Under capture the operator has no scratch and writes its fluxes in kernels of
    their own; a context's second call outside goes through the stage's kernels."""
    p = argon((17, 12, 9), dx=8e-6, seed=67)
    dt = stable_dt(p)
    st = StagState(p, "cuda")
    ctx = Context(p)
    ctx.init_state(st)
    ctx.rk3_step(st, dt, 0)
    nz = StepNoise(p, "cuda")
    ctx.fill_step_noise(nz, 1)
    names = [n for n in st.named(aux=True) if "flux" in n]
    for _ in range(2):
        for n in names:
            st.named(aux=True)[n].arr.fill_(-7.0)
        ctx.flux_stag(st, nz.face[0], nz.edge[0], nz.cen[0], dt)
    torch.cuda.synchronize()
    ref = st.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ctx.flux_stag(st, nz.face[0], nz.edge[0], nz.cen[0], dt)
    for n in names:
        st.named(aux=True)[n].arr.fill_(-7.0)
    g.replay()
    torch.cuda.synchronize()
    for n in names:
        a, r = st.named(aux=True)[n], ref.named(aux=True)[n]
        for c in range(r.ncomp):
            assert torch.equal(a.valid(c).cpu(), r.valid(c).cpu()), (n, c)
    ctx.close()
