"""GPU solvers through the C ABI against the oracle's restatement of the
reference solvers.  Every solve's true residual ||b - A x|| / ||b|| is
re-measured with the FP64 oracle operator."""
import numpy as np
import pytest

import leonardym_b200 as L
from leonardym_b200 import synth
from tests.helpers import CONFIGS, links_for, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["su3", "su2adj"])
def setup(request, oracle):
    name = request.param
    dims, rep, eps, kappa, csw = CONFIGS[name]
    links = links_for(name)
    lat = L.Lattice(dims, rep)
    gid = lat.upload(links)
    geom = oracle.Geometry(dims)
    b = synth.gaussian_spinor(dims, 3, 21)
    yield dict(dims=dims, rep=rep, kappa=kappa, csw=csw, links=links, lat=lat, gid=gid, geom=geom, b=b)
    lat.close()


def gpu_op(setup, cls, gamma5=True):
    op = cls(setup["lat"], setup["kappa"])
    if cls not in (L.DiracWilsonOperator, L.SquareDiracWilsonOperator):
        op.setCSW(setup["csw"])
    op.setGamma5(gamma5)
    op.setLattice(setup["gid"])
    return op


def true_res(oracle_op, b, x, shift=None):
    ax = oracle_op.multiply(x) if shift is None else oracle_op.multiply_add(x, x, shift)
    return float(np.linalg.norm(b - ax) / np.linalg.norm(b))


def test_cg_square_improved(setup, oracle):
    # ConjugateGradient on D^+D (configs: CG on D^dagger D to 1e-10 relative)
    b = setup["b"]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    cg = L.ConjugateGradient()
    cg.setPrecision(eps)
    cg.setMaximumSteps(5000)
    x = setup["lat"].new_vector()
    assert cg.solve(op, b, x)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    rc, xo, steps = oracle.cg(orc, b, eps, 5000)
    assert rc == 1
    assert abs(cg.getLastSteps() - steps) <= 2
    assert true_res(orc, b, x) < 1.5e-10
    assert rel(x, xo) < 1e-7


def test_bicgstab_square_improved(setup, oracle):
    b = setup["b"]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    s = L.BiConjugateGradient()
    s.setPrecision(eps)
    s.setMaximumSteps(5000)
    x = setup["lat"].new_vector()
    assert s.solve(op, b, x)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    rc, xo, steps = oracle.bicgstab(orc, b, eps, 5000)
    assert rc == 1
    # BiCGStab's trajectory depends on the summation order of its reductions: on the
    # ill-conditioned systems the iteration counts drift apart while both converge
    assert abs(s.getLastSteps() - steps) <= max(3, steps // 4)
    assert true_res(orc, b, x) < 1.5e-10
    assert rel(x, xo) < 1e-7


def test_bicgstab_shifted(setup, oracle):
    b = setup["b"]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    s = L.BiConjugateGradient()
    s.setPrecision(eps)
    s.setMaximumSteps(5000)
    x = setup["lat"].new_vector()
    assert s.solve(op, b, x, shift=0.05)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    assert true_res(orc, b, x, 0.05) < 1.5e-10


@pytest.mark.parametrize("gamma5", [False, True])
def test_preconditioned_bicgstab(setup, gamma5, oracle):
    b = setup["b"]
    prec = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.ImprovedDiracWilsonOperator, gamma5)
    s = L.PreconditionedBiCGStab()
    s.setPrecision(prec)
    s.setMaximumSteps(5000)
    x = setup["lat"].new_vector()
    assert s.solve(op, b, x)
    orc = oracle.Operator(setup["geom"], setup["links"], "Improved", setup["kappa"], setup["csw"], gamma5)
    rc, xo, steps = oracle.preconditioned_bicgstab(orc, b, prec, 5000)
    assert rc == 1
    assert abs(s.getLastSteps() - steps) <= max(3, steps // 4)
    # the even-odd path solves D x = b (gamma5 = false operator) whatever the flag
    D = oracle.Operator(setup["geom"], setup["links"], "Improved", setup["kappa"], setup["csw"], False)
    assert true_res(D, b, x) < 1e-8
    assert rel(x, xo) < 1e-7


@pytest.mark.parametrize("mode", ["double", "single", "half"])
def test_even_odd_cg_true_residual(setup, mode, oracle):
    b = setup["b"]
    op = gpu_op(setup, L.ImprovedDiracWilsonOperator, False)
    s = L.EvenOddConjugateGradient(mode, 1e-10)
    x = setup["lat"].new_vector()
    assert s.solve(op, b, x)
    D = oracle.Operator(setup["geom"], setup["links"], "Improved", setup["kappa"], setup["csw"], False)
    r = true_res(D, b, x)
    assert r <= 1e-10
    assert s.stats.true_residual <= 1e-10
    assert abs(s.stats.true_residual - r) < 1e-11


@pytest.mark.parametrize("mode", ["single", "half"])
@pytest.mark.parametrize("cls", ["Improved", "DiracWilson"])
def test_even_odd_bicgstab_mixed_true_residual(setup, mode, cls, oracle):
    b = setup["b"]
    gcls = L.ImprovedDiracWilsonOperator if cls == "Improved" else L.DiracWilsonOperator
    op = gpu_op(setup, gcls, False)
    s = L.EvenOddBiCGStab(mode, 1e-10)
    x = setup["lat"].new_vector()
    assert s.solve(op, b, x), s.stats.as_dict()
    csw = setup["csw"] if cls == "Improved" else 0.0
    D = oracle.Operator(setup["geom"], setup["links"], cls, setup["kappa"], csw, False)
    r = true_res(D, b, x)
    assert r <= 1e-10
    assert abs(s.stats.true_residual - r) < 1e-11
    assert s.stats.reliable_updates >= 1


def test_even_odd_bicgstab_rejects_guess(setup):
    op = gpu_op(setup, L.ImprovedDiracWilsonOperator, False)
    s = L.EvenOddBiCGStab("single", 1e-10)
    x = setup["lat"].new_vector()
    with pytest.raises(L.LymError):
        s.solve(op, setup["b"], x, initial_guess=setup["b"])


def test_even_odd_cg_wilson(setup, oracle):
    b = setup["b"]
    op = gpu_op(setup, L.DiracWilsonOperator, False)
    s = L.EvenOddConjugateGradient("single", 1e-10)
    x = setup["lat"].new_vector()
    assert s.solve(op, b, x)
    D = oracle.Operator(setup["geom"], setup["links"], "DiracWilson", setup["kappa"], 0.0, False)
    assert true_res(D, b, x) <= 1e-10


def test_multishift_mass_estrapolation(setup, oracle):
    b = setup["b"]
    shifts = [0.5, 0.1, 0.01]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    ms = L.MultishiftSolver.getInstance("mass_estrapolation")
    ms.setPrecision(eps)
    sols = []
    assert ms.solve(op, b, sols, shifts)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    rc, osols, _ = oracle.me_multishift(orc, b, shifts, eps)
    for x, xo, s in zip(sols, osols, shifts):
        assert true_res(orc, b, x, s) < 1.5e-10
        assert rel(x, xo) < 1e-7


def test_multishift_cg(setup, oracle):
    b = setup["b"]
    shifts = list(np.logspace(-4, 0, 12))
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    ms = L.MultishiftSolver.getInstance("multishift_cg")
    ms.setPrecision(eps)
    ms.setMaxSteps(10000)
    sols = []
    assert ms.solve(op, b, sols, shifts)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    for x, s in zip(sols, shifts):
        assert true_res(orc, b, x, s) < 3e-10


def test_multishift_minimal_residual(setup, oracle):
    # MMMRMultishiftSolver: base system = last shift; negative shifts by separate CG
    b = setup["b"]
    shifts = [-0.001, 0.5, 0.1, 0.02]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    ms = L.MultishiftSolver.getInstance("minimal_residual")
    ms.setPrecision(eps)
    ms.setMaxSteps(10000)
    sols = []
    assert ms.solve(op, b, sols, shifts)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    rc, osols, steps = oracle.mmmr_multishift(orc, b, shifts, eps, 10000)
    assert rc == 1
    for x, xo, s in zip(sols, osols, shifts):
        assert true_res(orc, b, x, s) < 2e-10
        assert rel(x, xo) < 1e-7


@pytest.mark.parametrize("l", [2, 4])
def test_bicgstab_l_matches_oracle(setup, l, oracle):
    # BiConjugateGradient::solve(dirac, source, solution, int l) (BiConjugateGradient.cpp:130-317)
    b = setup["b"]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    rc, xo, steps = oracle.bicgstab_l(orc, l, b, eps, 3000)
    s = L.BiConjugateGradient()
    s.setPrecision(eps)
    s.setMaximumSteps(3000)
    x = setup["lat"].new_vector()
    ok = s.solve(gpu_op(setup, L.SquareImprovedDiracWilsonOperator), b, x, l=l)
    if rc != 1:  # the algorithm does not converge on this system in the oracle either
        assert not ok or true_res(orc, b, x) < 1.5e-10
        return
    assert ok
    # BiCGStab(l)'s iteration count follows rounding closely on these systems (two
    # FP64 implementations with different summation orders differ by tens of percent), so the
    # checked properties are convergence, the true residual and the solution
    assert s.getLastSteps() <= 2 * steps + 10
    assert true_res(orc, b, x) < 1.5e-10
    assert rel(x, xo) < 1e-7


def test_bicgstab_preconditioned_matches_oracle(setup, oracle):
    # BiConjugateGradient::solve(dirac, source, solution, preconditioner) (BiConjugateGradient.cpp:11-128)
    b = setup["b"]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    orc = oracle.Operator(setup["geom"], setup["links"], "Improved", setup["kappa"], setup["csw"], False)
    pre_o = oracle.Operator(setup["geom"], setup["links"], "DiracWilson", 0.05, 0.0, False)
    rc, xo, steps = oracle.bicgstab_precond(orc, pre_o, b, eps, 3000)
    pre = L.DiracWilsonOperator(setup["lat"], 0.05)
    pre.setGamma5(False)
    pre.setLattice(setup["gid"])
    s = L.BiConjugateGradient()
    s.setPrecision(eps)
    s.setMaximumSteps(3000)
    x = setup["lat"].new_vector()
    ok = s.solve(gpu_op(setup, L.ImprovedDiracWilsonOperator, False), b, x, preconditioner=pre)
    assert ok == (rc == 1)
    if rc == 1:
        assert abs(s.getLastSteps() - steps) <= max(3, steps // 4)
        assert rel(x, xo) < 1e-7


def test_multishift_chronological(setup, oracle):
    # ChronologicalMultishiftSolver (ChronologicalMultishiftSolver.cpp:11-194): the second solve
    # starts every shift from the first solve's solutions (the chronological guesses)
    b = setup["b"]
    shifts = [0.5, 0.1, 0.01]
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareImproved", setup["kappa"], setup["csw"], True)
    ms = L.MultishiftSolver.getInstance("chronological_mass_estrapolation")
    ms.setPrecision(eps)
    sols = []
    assert ms.solve(op, b, sols, shifts)
    first_iters = ms.stats.iterations
    rc, osols = oracle.chrono_multishift(orc, b, shifts, eps)
    assert rc == 1
    for x, xo, s in zip(sols, osols, shifts):
        assert true_res(orc, b, x, s) < 1.5e-10
        assert rel(x, xo) < 1e-7
    b2 = b + 1e-3 * synth.gaussian_spinor(setup["dims"], 3, 22)
    sols2 = []
    assert ms.solve(op, b2, sols2, shifts)
    rc, osols2 = oracle.chrono_multishift(orc, b2, shifts, eps, previous=osols)
    for x, xo, s in zip(sols2, osols2, shifts):
        assert true_res(orc, b2, x, s) < 1.5e-10
        assert rel(x, xo) < 1e-7
    assert ms.stats.iterations < first_iters


@pytest.mark.parametrize("mode", ["single", "half"])
def test_multishift_cg_mixed(setup, oracle, mode):
    # RHMC multishift on the squared even-odd operator: FP32 / FP16 inner storage, FP64
    # recurrences; every shift's FP64 true residual <= 1e-10 and the solutions equal the
    # oracle's FP64 mass-estrapolation solutions
    b = setup["b"]
    shifts = list(np.logspace(-4, 0, 12))
    eps = (1e-10) ** 2 * float(np.vdot(b, b).real)
    op = gpu_op(setup, L.SquareEvenOddImprovedDiracWilsonOperator)
    ms = L.MultishiftSolver.getInstance(f"multishift_cg_mixed_{mode}")
    ms.setPrecision(eps)
    ms.setMaxSteps(10000)
    sols = []
    assert ms.solve(op, b, sols, shifts)
    assert ms.stats.true_residual <= 1e-10
    assert ms.stats.reliable_updates >= 1
    orc = oracle.Operator(setup["geom"], setup["links"], "SquareEvenOddImproved", setup["kappa"], setup["csw"],
                          True)
    rc, osols, _ = oracle.me_multishift(orc, b, shifts, eps, 10000)
    assert rc == 1
    for x, xo, s in zip(sols, osols, shifts):
        assert true_res(orc, b, x, s) <= 1.05e-10
        assert rel(x, xo) < 1e-7


def test_multishift_cg_mixed_needs_rhmc_operator(setup):
    op = gpu_op(setup, L.SquareImprovedDiracWilsonOperator)
    ms = L.MultishiftSolver.getInstance("multishift_cg_mixed_single")
    with pytest.raises(L.LymError):
        ms.solve(op, setup["b"], [], [0.1, 0.01])
    op = gpu_op(setup, L.SquareEvenOddImprovedDiracWilsonOperator)
    with pytest.raises(L.LymError):
        ms.solve(op, setup["b"], [], [-1.0, 0.01])


@pytest.mark.parametrize("kind,alg", [("SquareImproved", "mass_estrapolation"),
                                      ("SquareImproved", "minimal_residual"),
                                      ("SquareEvenOddImproved", "mass_estrapolation"),
                                      ("SquareEvenOddImproved", "multishift_cg_mixed_half")])
def test_rational_evaluate(setup, oracle, kind, alg):
    # RationalApproximation::evaluate: sum_i alpha_i (A + beta_i)^{-1} b, against the oracle's
    # restatement (FP64 mass-estrapolation multishift)
    b = setup["b"]
    alphas, betas = [0.31, 0.12, 0.047, 0.011], [0.9, 0.17, 0.03, 0.004]
    eps = (1e-11) ** 2 * float(np.vdot(b, b).real)
    cls = L.SquareImprovedDiracWilsonOperator if kind == "SquareImproved" else L.SquareEvenOddImprovedDiracWilsonOperator
    ra = L.RationalApproximation(alphas, betas, L.MultishiftSolver.getInstance(alg))
    ra.setPrecision(eps)
    ra.setMaximumRecursion(10000)
    out = setup["lat"].new_vector()
    ra.evaluate(gpu_op(setup, cls), out, b)
    orc = oracle.Operator(setup["geom"], setup["links"], kind, setup["kappa"], setup["csw"], True)
    rc, ref = oracle.rational_evaluate(orc, alphas, betas, b, eps, 10000)
    assert rc == 1
    assert rel(out, ref) < 1e-8
    assert abs(ra.evaluate(0.25) - oracle.rational_value(alphas, betas, 0.25)) < 1e-14


def test_rhmc_action_energy_and_force_solves(setup, oracle):
    # NFlavorFermionAction: energy = sum_k Re <phi_k, r_k(A) phi_k>; updateForce's solves
    # x_i = (A + beta_i)^{-1} phi, y_i = D x_i, on the even-odd RHMC operator
    b = setup["b"]
    phi2 = synth.gaussian_spinor(setup["dims"], 3, 23)
    approx = [([0.31, 0.12, 0.047], [0.9, 0.17, 0.03]), ([0.5, 0.2], [0.4, 0.05])]
    eps = (1e-11) ** 2 * float(np.vdot(b, b).real)
    sq = gpu_op(setup, L.SquareEvenOddImprovedDiracWilsonOperator)
    D = gpu_op(setup, L.EvenOddImprovedDiracWilsonOperator)
    ras = []
    for al, be in approx:
        ms = L.MultishiftSolver.getInstance("mass_estrapolation")
        ms.setPrecision(eps)
        ms.setMaxSteps(10000)
        ra = L.RationalApproximation(al, be, ms)
        ra.setPrecision(eps)
        ra.setMaximumRecursion(10000)
        ras.append(ra)
    act = L.NFlavorFermionAction(D, sq, ras)
    act.addPseudoFermion(b)
    act.addPseudoFermion(phi2)
    A = oracle.Operator(setup["geom"], setup["links"], "SquareEvenOddImproved", setup["kappa"], setup["csw"], True)
    Do = oracle.Operator(setup["geom"], setup["links"], "EvenOddImproved", setup["kappa"], setup["csw"], True)
    e_ref = oracle.rhmc_energy(A, approx, [b, phi2], eps, 10000)
    assert abs(act.energy() - e_ref) <= 1e-9 * abs(e_ref)
    Xs, Ys = act.solves()
    for (al, be), phi, X, Y in zip(approx, [b, phi2], Xs, Ys):
        rc, xo, yo = oracle.rhmc_force_solves(A, Do, be, phi, eps, 10000)
        assert rc == 1
        for x, y, xr, yr in zip(X, Y, xo, yo):
            assert rel(x, xr) < 1e-8
            assert rel(y, yr) < 1e-8


@pytest.mark.parametrize("rep", ["su3", "su2adj"])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 6, 2, 6), (4, 4, 2, 10), (4, 4, 4, 6)])
@pytest.mark.parametrize("kind", ["SquareDiracWilson", "SquareImproved", "SquareEvenOddImproved"])
def test_fused_square_cg(rep, dims, kind, oracle):
    """CG on the squared operators, whose vector work runs inside the products (Wilson and clover:
    the whole solve in one launch): fewer half-sites than a block, ragged last blocks, a shift, and
    more iterations than one launch runs."""
    kappa, csw = (0.12, 1.0) if rep == "su3" else (0.15, 1.2)
    links = synth.fermion_links(dims, rep, 0.3, 71)
    lat = L.Lattice(dims, rep)
    try:
        cls = {"SquareDiracWilson": L.SquareDiracWilsonOperator, "SquareImproved": L.SquareImprovedDiracWilsonOperator,
               "SquareEvenOddImproved": L.SquareEvenOddImprovedDiracWilsonOperator}[kind]
        op = cls(lat)
        op.setKappa(kappa)
        clover = kind != "SquareDiracWilson"
        if clover:
            op.setCSW(csw)
        op.setLattice(lat.upload(links))
        orc = oracle.Operator(oracle.Geometry(dims), links, kind, kappa, csw if clover else 0.0, True)
        b = synth.gaussian_spinor(dims, 3, 72)
        eps = 1e-22 * float(np.vdot(b, b).real)
        cg = L.ConjugateGradient()
        cg.setPrecision(eps)
        x = lat.new_vector()
        assert cg.solve(op, b, x)
        rc, xo, steps = oracle.cg(orc, b, eps, 3000)
        assert abs(cg.getLastSteps() - steps) <= 2
        assert rel(x, xo) < 1e-9 and rel(orc.multiply(x), b) < 1.1e-11
        # one step of the reference, then a run past the iterations of a launch (no stop)
        cg.setMaximumSteps(1)
        cg.setPrecision(0.0)
        assert not cg.solve(op, b, x)
        assert rel(x, oracle.cg(orc, b, 0.0, 1)[1]) < 1e-12
        if dims == (4, 4, 4, 6) and kind != "SquareEvenOddImproved":  # |r|^2 stays above 1e-150
            cg.setMaximumSteps(530)
            assert not cg.solve(op, b, x) and cg.stats.iterations == 530
            assert rel(orc.multiply(x), b) < 1e-12
        # with shifts, one CG each
        ms = L.MultishiftSolver.getInstance("mass_estrapolation")
        ms.setPrecision(eps)
        sols = []
        assert ms.solve(op, b, sols, [0.0, 0.3])
        assert rel(orc.multiply(sols[1]) + 0.3 * sols[1], b) < 1.1e-11
    finally:
        lat.close()


@pytest.mark.parametrize("rep,dims,kind", [
    ("su3", (2, 2, 2, 2), "SquareEvenOddImproved"), ("su2adj", (2, 6, 2, 10), "SquareEvenOddImproved"),
    ("su3", (2, 2, 2, 2), "SquareDiracWilson"), ("su3", (4, 4, 2, 10), "SquareImproved"),
    ("su2adj", (4, 4, 4, 6), "SquareImproved"), ("su3", (4, 4, 4, 6), "SquareDiracWilson"),
    ("su3", (8, 8, 8, 74), "SquareEvenOddImproved"), ("su3", (8, 8, 8, 76), "SquareEvenOddImproved")])
def test_one_launch_multishift(rep, dims, kind, oracle):
    """The FP64 multishift in one launch: ragged and single tiles, either side of the size from which
    its steps are launches again, step counts around the window of 8, more steps than one launch runs."""
    kappa, csw = (0.12, 1.0) if rep == "su3" else (0.15, 1.2)
    links = synth.fermion_links(dims, rep, 0.3, 81)
    lat = L.Lattice(dims, rep)
    try:
        op = {"SquareDiracWilson": L.SquareDiracWilsonOperator, "SquareImproved": L.SquareImprovedDiracWilsonOperator,
              "SquareEvenOddImproved": L.SquareEvenOddImprovedDiracWilsonOperator}[kind](lat)
        op.setKappa(kappa)
        clover = kind != "SquareDiracWilson"
        if clover:
            op.setCSW(csw)
        op.setLattice(lat.upload(links))
        orc = oracle.Operator(oracle.Geometry(dims), links, kind, kappa, csw if clover else 0.0, True)
        b = synth.gaussian_spinor(dims, 3, 82)
        eps = 1e-22 * float(np.vdot(b, b).real)
        ms = L.MultishiftSolver.getInstance("multishift_cg")
        ms.setMaxSteps(3000)
        ms.setPrecision(eps)
        shifts, sols = [0.3, 0.02, 1e-3, 0.0, 2.0], []
        assert ms.solve(op, b, sols, shifts)
        for x, s in zip(sols, shifts):
            assert rel(orc.multiply(x) + s * x, b) < 5e-11
        if lat.V > 1000:
            return
        # k steps give the base system's k-th CG iterate, whatever the place within a window
        ms.setPrecision(0.0)
        for k in (1, 7, 8, 9):
            ms.setMaxSteps(k)
            assert not ms.solve(op, b, sols, shifts) and ms.stats.iterations == k
            assert rel(sols[3], oracle.cg(orc, b, 0.0, k, guess=np.zeros_like(b))[1]) < 1e-11
        if dims == (4, 4, 4, 6):  # |r|^2 and the shift's zeta stay far from underflow
            ms.setMaxSteps(530)
            assert not ms.solve(op, b, sols[:2], [0.0, 1e-6]) and ms.stats.iterations == 530
            assert rel(orc.multiply(sols[0]), b) < 1e-12
    finally:
        lat.close()


def test_one_launch_solvers_of_two_threads(oracle):
    """A CG and a multishift, each in one launch and on a context of its own, from two threads at
    once: their grids would not fit on the GPU together, so they take turns."""
    import threading

    kappa, csw = 0.12, 1.0
    jobs, errors = [], []
    for dims, kind, cls in (((8, 8, 8, 8), "SquareImproved", L.SquareImprovedDiracWilsonOperator),
                            ((8, 8, 8, 74), "SquareEvenOddImproved", L.SquareEvenOddImprovedDiracWilsonOperator)):
        links = synth.fermion_links(dims, "su3", 0.3, 91)
        lat = L.Lattice(dims, "su3")
        op = cls(lat, kappa, csw)
        op.setLattice(lat.upload(links))
        b = synth.gaussian_spinor(dims, 3, 92)
        orc = oracle.Operator(oracle.Geometry(dims), links, kind, kappa, csw, True)
        jobs.append((lat, op, b, orc, 1e-22 * float(np.vdot(b, b).real)))
    (lat_a, op_a, b_a, orc_a, eps_a), (lat_b, op_b, b_b, orc_b, eps_b) = jobs
    x, sols = lat_a.new_vector(), []

    def run_cg():
        cg = L.ConjugateGradient()
        cg.setPrecision(eps_a)
        for _ in range(40):
            if not cg.solve(op_a, b_a, x):
                errors.append("cg")

    def run_multishift():
        ms = L.MultishiftSolver.getInstance("multishift_cg")
        ms.setPrecision(eps_b)
        for _ in range(6):
            if not ms.solve(op_b, b_b, sols, [0.0, 0.3]):
                errors.append("multishift")

    def guarded(f):
        try:
            f()
        except Exception as e:  # an error of the thread fails the test
            errors.append(e)

    try:
        threads = [threading.Thread(target=guarded, args=(f,)) for f in (run_cg, run_multishift)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors
        assert rel(orc_a.multiply(x), b_a) < 1.1e-11
        for y, s in zip(sols, (0.0, 0.3)):
            assert rel(orc_b.multiply(y) + s * y, b_b) < 5e-11
    finally:
        lat_a.close()
        lat_b.close()


@pytest.mark.parametrize("kind", ["SquareEvenOddImproved", "SquareImproved"])
def test_multishift_without_memory_for_its_window(kind, oracle):
    """Where there is no memory for the ring of residuals, the FP64 multishift updates its shifted
    vectors every step: the same iterates and solutions from ten vectors less.  (A solve with one
    shift first leaves 15 full vectors behind; four shifts take 11 without the ring.)"""
    dims, kappa, csw = (4, 4, 4, 6), 0.12, 1.0
    links = synth.fermion_links(dims, "su3", 0.3, 85)
    lat = L.Lattice(dims, "su3")
    lib = L.lib()
    try:
        op = {"SquareImproved": L.SquareImprovedDiracWilsonOperator,
              "SquareEvenOddImproved": L.SquareEvenOddImprovedDiracWilsonOperator}[kind](lat, kappa, csw)
        op.setLattice(lat.upload(links))
        orc = oracle.Operator(oracle.Geometry(dims), links, kind, kappa, csw, True)
        b = synth.gaussian_spinor(dims, 3, 86)
        eps = 1e-22 * float(np.vdot(b, b).real)
        ms = L.MultishiftSolver.getInstance("multishift_cg")

        def solve(shifts):
            sols, n = [], lib.lym_context_kernel_launches(lat.handle)
            ok = ms.solve(op, b, sols, shifts)
            return ok, sols, lib.lym_context_kernel_launches(lat.handle) - n

        shifts = [0.3, 0.02, 1e-3, 0.0]
        for eps_k, steps in ((eps, 3000), (0.0, 1), (0.0, 7), (0.0, 8), (0.0, 9)):
            lib.lym_context_trim(lat.handle)
            ms.setPrecision(eps)
            ms.setMaxSteps(3000)
            one = solve([0.0])[2]
            ms.setPrecision(eps_k)
            ms.setMaxSteps(steps)
            try:
                assert lib.lym_context_inject_alloc_failures(lat.handle, 1000) == 0
                ok, sols, launches = solve(shifts)
            finally:
                lib.lym_context_inject_alloc_failures(lat.handle, 0)
            assert launches > one + 8  # not the one-launch form
            if eps_k > 0.0:
                assert ok
                for x, s in zip(sols, shifts):
                    assert rel(orc.multiply(x) + s * x, b) < 5e-11
            else:
                assert not ok and ms.stats.iterations == steps
                xo = oracle.cg(orc, b, 0.0, steps, guess=np.zeros_like(b))[1]
                assert rel(sols[3], xo) < 1e-11
            again = solve(shifts)[1]  # with memory: the window's updates
            for x, y in zip(sols, again):
                assert rel(x, y) < (1e-9 if ok else 1e-11)
    finally:
        lat.close()


# CG on the squared kinds takes one launch of 2 blocks per SM up to 148 * 64 = 9472 sites, of 4 up to
# 18944, and launches per iteration above; the FP64 multishift one launch up to 37888 sites.
@pytest.mark.parametrize("rep", ["su3", "su2adj"])
@pytest.mark.parametrize("dims", [(8, 8, 8, 18), (8, 8, 8, 20), (6, 8, 14, 28), (8, 8, 8, 38)])
@pytest.mark.parametrize("kind", ["SquareDiracWilson", "SquareImproved"])
def test_square_cg_of_every_size(rep, dims, kind, oracle):
    kappa, csw = (0.12, 1.0) if rep == "su3" else (0.15, 1.2)
    lat, op, orc = _square_operator(dims, rep, kind, kappa, csw, 95, oracle)
    try:
        b = synth.gaussian_spinor(dims, 3, 96)
        eps = 1e-22 * float(np.vdot(b, b).real)
        cg = L.ConjugateGradient()
        cg.setPrecision(eps)
        x, n = lat.new_vector(), L.lib().lym_context_kernel_launches(lat.handle)
        assert cg.solve(op, b, x)
        n = L.lib().lym_context_kernel_launches(lat.handle) - n
        assert (n < cg.stats.iterations) == (lat.V <= 18944)
        assert rel(orc.multiply(x), b) < 1.1e-11
        cg.setPrecision(0.0)
        for k in (1, 6):
            cg.setMaximumSteps(k)
            assert not cg.solve(op, b, x)
            assert rel(x, oracle.cg(orc, b, 0.0, k)[1]) < 1e-12
        # with a shift, from the guess of the solver that starts at the previous shift's solution
        ms = L.MultishiftSolver.getInstance("mass_estrapolation")
        ms.setPrecision(eps)
        sols = []
        assert ms.solve(op, b, sols, [0.05, 0.3])
        for y, s in zip(sols, (0.05, 0.3)):
            assert rel(orc.multiply(y) + s * y, b) < 1.1e-11
    finally:
        lat.close()


@pytest.mark.parametrize("rep,dims,kind", [
    ("su3", (8, 8, 8, 40), "SquareImproved"), ("su2adj", (8, 8, 8, 40), "SquareDiracWilson"),
    ("su3", (8, 8, 8, 74), "SquareImproved"), ("su2adj", (8, 8, 8, 74), "SquareImproved"),
    ("su3", (8, 8, 8, 76), "SquareImproved"), ("su2adj", (8, 8, 8, 76), "SquareDiracWilson"),
    ("su2adj", (8, 8, 8, 74), "SquareEvenOddImproved"), ("su2adj", (8, 8, 8, 76), "SquareEvenOddImproved")])
def test_multishift_of_every_size(rep, dims, kind, oracle):
    """Blocks that walk one tile or several, and launches per step, whose steps around the window of
    8 are checked against the oracle's."""
    kappa, csw = (0.12, 1.0) if rep == "su3" else (0.15, 1.2)
    lat, op, orc = _square_operator(dims, rep, kind, kappa, csw, 97, oracle)
    try:
        b = synth.gaussian_spinor(dims, 3, 98)
        eps = 1e-22 * float(np.vdot(b, b).real)
        ms = L.MultishiftSolver.getInstance("multishift_cg")
        ms.setMaxSteps(3000)
        ms.setPrecision(eps)
        shifts, sols, n = [0.3, 1e-3, 0.0], [], L.lib().lym_context_kernel_launches(lat.handle)
        assert ms.solve(op, b, sols, shifts)
        n = L.lib().lym_context_kernel_launches(lat.handle) - n
        assert (n < ms.stats.iterations) == (lat.V <= 37888)
        for x, s in zip(sols, shifts):
            assert rel(orc.multiply(x) + s * x, b) < 5e-11
        ms.setPrecision(0.0)
        for k in (7, 8, 9):
            ms.setMaxSteps(k)
            assert not ms.solve(op, b, sols, shifts) and ms.stats.iterations == k
            assert rel(sols[2], oracle.cg(orc, b, 0.0, k, guess=np.zeros_like(b))[1]) < 1e-11
    finally:
        lat.close()


def _square_operator(dims, rep, kind, kappa, csw, seed, oracle):
    links = synth.fermion_links(dims, rep, 0.3, seed)
    lat = L.Lattice(dims, rep)
    op = {"SquareDiracWilson": L.SquareDiracWilsonOperator, "SquareImproved": L.SquareImprovedDiracWilsonOperator,
          "SquareEvenOddImproved": L.SquareEvenOddImprovedDiracWilsonOperator}[kind](lat)
    op.setKappa(kappa)
    clover = kind != "SquareDiracWilson"
    if clover:
        op.setCSW(csw)
    op.setLattice(lat.upload(links))
    return lat, op, oracle.Operator(oracle.Geometry(dims), links, kind, kappa, csw if clover else 0.0, True)
