"""The structure factor's routes: more variables than a block's shared memory holds
(13 and up) and the input transformed in place or packed first, odd and even half
spectra, against the NumPy restatement within 1e-12 (the FFT libraries' rounding, as in
the tests of the default route)."""
import numpy as np
import pytest
import torch

from fhdex_b200.fab import CELL, MultiFab
from fhdex_b200.structfact import StructFact
from oracle.structfact import StructFactOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvar", [12, 13])
@pytest.mark.parametrize("shape_xyz,ng", [((6, 4, 5), 0), ((7, 3, 4), 1), ((2, 6, 3), 0)])
def test_routes_match_oracle(nvar, shape_xyz, ng):
    rng = np.random.default_rng(17)
    ncov = nvar * (nvar + 1) // 2
    scaling = list(rng.uniform(0.5, 2.0, ncov))
    sf = StructFact(shape_xyz, [f"v{i}" for i in range(nvar)], scaling)
    zyx = shape_xyz[::-1]
    ora = StructFactOracle(zyx, nvar, scaling)
    mf = MultiFab(shape_xyz, CELL, nvar, ng, device="cuda")
    for _ in range(2):
        v = rng.standard_normal((nvar,) + zyx)
        mf.valid().copy_(torch.from_numpy(v))
        sf.fort_structure(mf)
        ora.fort_structure(v)
    for zero_avg in (0, 1):
        got = [m.valid().cpu().numpy() for m in sf.finalize(zero_avg)]
        for g, r in zip(got, ora.finalize(zero_avg)):
            assert np.abs(g - r).max() < 1e-12 * max(np.abs(r).max(), 1e-300)
    sf.close()


@pytest.mark.parametrize("shape_xyz", [(6, 4, 5), (7, 3, 4)])
def test_auto_pairs_have_positive_zero_imaginary_parts(shape_xyz):
    """A variable with itself: the imaginary part is +0.0 at every point, the mirrored
    ones too, as where each point's own products are subtracted."""
    sf = StructFact(shape_xyz, ["a"], [1.0])
    mf = MultiFab(shape_xyz, CELL, 1, 0, device="cuda")
    mf.valid().copy_(torch.randn((1,) + shape_xyz[::-1], dtype=torch.float64, generator=torch.Generator().manual_seed(19)))
    sf.fort_structure(mf)
    im = sf.finalize()[1].valid(0)
    assert (im == 0).all() and not torch.signbit(im).any()
    sf.close()


def test_pair_list_with_more_variables_than_pairs():
    """Two pairs of four variables: one variable at a time through the transform, in no more
    memory than two full grids per pair, the four half spectra and one dense copy, and the
    same result as the two pairs each by itself (within the FFT's rounding: a plan of one
    transform against one of two)."""
    shape = (128, 120, 124)
    cells, half = 128 * 120 * 124, 65 * 120 * 124
    mf = MultiFab(shape, CELL, 4, 0, device="cuda")
    mf.valid().copy_(torch.randn((4,) + shape[::-1], dtype=torch.float64, generator=torch.Generator().manual_seed(20)))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    sf = StructFact(shape, list("abcd"), [1.0, 2.0], pairs=([0, 2], [1, 3]))
    # (each of the allocations is rounded up to 2 MiB)
    assert free - torch.cuda.mem_get_info()[0] <= 8 * (2 * 2 * cells + 4 * 2 * half + cells) + 6 * 2 ** 21
    for _ in range(2):
        sf.fort_structure(mf)
    got = sf.finalize()
    sf.close()
    for c, (a, b) in enumerate([(0, 1), (2, 3)]):
        one = StructFact(shape, list("abcd"), [1.0 + c], pairs=([a], [b]))
        for _ in range(2):
            one.fort_structure(mf)
        for g, w in zip(got, one.finalize()):
            assert (g.valid(c) - w.valid(0)).abs().max() < 1e-12 * w.valid(0).abs().max(), c
        one.close()


def test_outputs_of_more_than_2_31_values():
    """1030 pairs at 128^3 are 2.16e9 values per output, with the components from 1024 on
    beyond 32-bit offsets (about 70 GB in all).  Every pair is the same one."""
    shape, ncov = (128, 128, 128), 1030
    mf = MultiFab(shape, CELL, 2, 0, device="cuda")
    mf.valid().copy_(torch.randn((2,) + shape, dtype=torch.float64, generator=torch.Generator().manual_seed(18)))
    one = StructFact(shape, ["a", "b"], [1.0], pairs=([1], [0]))
    many = StructFact(shape, ["a", "b"], [1.0] * ncov, pairs=([1] * ncov, [0] * ncov))
    for sf in (one, many):
        sf.fort_structure(mf)
    want, got = one.finalize(), many.finalize()
    for g, w in zip(got, want):
        for c in (0, 511, 1023, 1024, 1029):
            assert torch.equal(g.valid(c), w.valid(0)), c
    del got, g
    one.close()
    many.close()
    torch.cuda.empty_cache()
