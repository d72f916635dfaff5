"""Many right-hand sides through the batched stencil (lym_solve_block): every result
meets the 1e-10 true residual re-measured with the FP64 oracle operator, and equals
the same source solved alone within what the 1e-10 residual allows."""
import numpy as np
import pytest

import leonardym_b200 as L
from leonardym_b200 import synth
from tests.helpers import CONFIGS, links_for, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["su3", "su2adj"])
def setup(request, oracle):
    dims, rep, eps, kappa, csw = CONFIGS[request.param]
    links = links_for(request.param)
    lat = L.Lattice(dims, rep)
    op = L.ImprovedDiracWilsonOperator(lat, kappa, csw, gamma5=False)
    op.setLattice(links)
    D = oracle.Operator(oracle.Geometry(dims), links, "Improved", kappa, csw, False)
    srcs = [synth.point_source(dims, 3, a, 1) for a in range(2)] + \
           [synth.z2_source(dims, 3, 5, stream=(1 << 21) + k) for k in range(2)] + \
           [synth.gaussian_spinor(dims, 3, 40 + k) for k in range(2)]
    yield dict(lat=lat, op=op, D=D, srcs=srcs)
    lat.close()


SOLVERS = {"cg": L.EvenOddConjugateGradient, "bicgstab": L.EvenOddBiCGStab}


@pytest.mark.parametrize("algo", ["cg", "bicgstab"])
@pytest.mark.parametrize("mode", ["single", "half"])
@pytest.mark.parametrize("batch", [2, 8])
def test_block_solve_alone_and_in_the_mix(setup, algo, mode, batch):
    s = SOLVERS[algo](mode, 1e-10)
    ok, sols = s.solve_block(setup["op"], setup["srcs"], batch=batch)
    assert ok
    for j, (b, x) in enumerate(zip(setup["srcs"], sols)):
        r = np.linalg.norm(b - setup["D"].multiply(x)) / np.linalg.norm(b)
        assert r <= 1e-10, (j, r)
        assert s.block_stats[j].true_residual <= 1e-10
        alone = setup["lat"].new_vector()
        single = SOLVERS[algo](mode, 1e-10)
        assert single.solve(setup["op"], b, alone)
        assert rel(x, alone) < 1e-8


def test_block_rejects_bad_batch(setup):
    s = L.EvenOddConjugateGradient("single", 1e-10)
    with pytest.raises(L.LymError):
        s.solve_block(setup["op"], setup["srcs"], batch=3)


@pytest.mark.parametrize("minb", [19, 20, 36, 84])
def test_block_bicgstab_fused_omega_matches_separate_pass(setup, minb):
    """The staged stencil variants fold the BiCGStab omega sums into the epilogue of the
    t = S s launch; a direct variant keeps them in a separate pass.  Both meet the 1e-10
    true residual and agree, and the fused sums are added in a fixed order (a second
    solve repeats the first bit for bit)."""
    from leonardym_b200.dirac import set_batch_tile
    lat = setup["lat"]
    srcs = setup["srcs"]
    out = {}
    try:
        for variant in (minb, minb, 1):
            set_batch_tile(lat, 0, 0, variant)
            s = L.EvenOddBiCGStab("single", 1e-10)
            ok, sols = s.solve_block(setup["op"], srcs, batch=8)
            assert ok
            for j, (b, x) in enumerate(zip(srcs, sols)):
                r = np.linalg.norm(b - setup["D"].multiply(x)) / np.linalg.norm(b)
                assert r <= 1e-10, (variant, j, r)
            out.setdefault(variant, []).append((sols, [st.iterations for st in s.block_stats]))
    finally:
        set_batch_tile(lat, -1, 0)
    (a, ia), (b, ib) = out[minb]
    assert ia == ib
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    for x, y in zip(a, out[1][0][0]):
        assert rel(x, y) < 1e-8


@pytest.mark.parametrize("mode,decades", [("half", 1.6), ("single", 2.5)])
def test_block_reliable_updates_are_close_enough(oracle, mode, decades):
    """The recursion of a source runs over no more than 1.5 decades of the residual with FP16
    storage (2.5 with FP32) between updates from the FP64 residual: beyond that the solutions' error
    grows, by 4 % after two decades with FP16."""
    dims = (8, 8, 12, 16)
    lat = L.Lattice(dims, "su3")
    try:
        op = L.ImprovedDiracWilsonOperator(lat, 0.122, 1.7, gamma5=False)
        op.setLattice(synth.fermion_links(dims, "su3", 0.25, 33))
        srcs = [synth.gaussian_spinor(dims, 3, 200 + k) for k in range(16)]
        s = L.EvenOddBiCGStab(mode, 1e-10)
        ok, _ = s.solve_block(op, srcs, batch=16)
        assert ok
        # an update passes its threshold by part of an iteration's fall, the last one ends the solve
        assert np.mean([st.reliable_updates for st in s.block_stats]) >= 10.0 / decades - 0.6
    finally:
        lat.close()


def test_block_updates_go_on_without_memory(setup):
    """Identical sources all wait for their reliable update at once, and updates done together take a
    vector each: where no memory is left for these, the updates go one by one and the solve ends as
    ever.  (One step with all sources first, so that nothing else is left to allocate.)"""
    lat, b = setup["lat"], setup["srcs"][4]
    s = L.EvenOddBiCGStab("single", 1e-10)
    L.lib().lym_context_trim(lat.handle)
    s.maxSteps = 1
    assert not s.solve_block(setup["op"], [b] * 16, batch=16)[0]
    s.maxSteps = 20000
    held = L.lib().lym_context_device_bytes(lat.handle)
    try:
        assert L.lib().lym_context_inject_alloc_failures(lat.handle, 1000) == 0
        ok, sols = s.solve_block(setup["op"], [b] * 16, batch=16)
    finally:
        L.lib().lym_context_inject_alloc_failures(lat.handle, 0)
    assert ok
    for x in sols:
        assert np.linalg.norm(b - setup["D"].multiply(x)) <= 1e-10 * np.linalg.norm(b)
    assert L.lib().lym_context_device_bytes(lat.handle) == held
    # with memory the next solve does take the vectors
    assert s.solve_block(setup["op"], [b] * 16, batch=16)[0]
    assert L.lib().lym_context_device_bytes(lat.handle) > held
