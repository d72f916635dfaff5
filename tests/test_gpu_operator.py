"""GPU parity of the operator application against the oracle (through the C ABI).

Bar: FP64 stencil within 1e-13 relative of the oracle, FP32 within 1e-6, FP16
within 1e-2 (storage precision 2^-11 with per-site norms); layout tables bit-exact.
"""
import numpy as np
import pytest

import leonardym_b200 as L
from leonardym_b200 import synth
from tests.helpers import CONFIGS, links_for, rel

pytestmark = pytest.mark.gpu

KINDS = ["DiracWilson", "Improved", "EvenOddImproved", "SquareDiracWilson", "SquareImproved",
         "SquareEvenOddImproved"]
GPU_CLASS = {
    "DiracWilson": L.DiracWilsonOperator, "Improved": L.ImprovedDiracWilsonOperator,
    "EvenOddImproved": L.EvenOddImprovedDiracWilsonOperator, "SquareDiracWilson": L.SquareDiracWilsonOperator,
    "SquareImproved": L.SquareImprovedDiracWilsonOperator,
    "SquareEvenOddImproved": L.SquareEvenOddImprovedDiracWilsonOperator,
}


@pytest.fixture(scope="module", params=["su3", "su2adj"])
def setup(request, oracle):
    name = request.param
    dims, rep, eps, kappa, csw = CONFIGS[name]
    links = links_for(name)
    lat = L.Lattice(dims, rep)
    gid = lat.upload(links)
    geom = oracle.Geometry(dims)
    yield dict(name=name, dims=dims, rep=rep, kappa=kappa, csw=csw, links=links, lat=lat, gid=gid, geom=geom)
    lat.close()


def make(setup, kind, gamma5, oracle):
    gpu = GPU_CLASS[kind](setup["lat"])
    gpu.setKappa(setup["kappa"])
    if kind not in ("DiracWilson", "SquareDiracWilson"):
        gpu.setCSW(setup["csw"])
    gpu.setGamma5(gamma5)
    gpu.setLattice(setup["gid"])
    csw = 0.0 if "Wilson" in kind else setup["csw"]
    orc = oracle.Operator(setup["geom"], setup["links"], kind, setup["kappa"], csw, gamma5)
    return gpu, orc


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("gamma5", [True, False])
def test_multiply_matches_oracle(setup, kind, gamma5, oracle):
    gpu, orc = make(setup, kind, gamma5, oracle)
    x = synth.gaussian_spinor(setup["dims"], 3, 7)
    out = setup["lat"].new_vector()
    gpu.multiply(out, x)
    assert rel(out, orc.multiply(x)) < 1e-13


@pytest.mark.parametrize("kind", ["DiracWilson", "Improved", "SquareDiracWilson", "SquareImproved",
                                  "SquareEvenOddImproved"])
@pytest.mark.parametrize("gamma5", [True, False])
def test_multiply_add_matches_oracle(setup, kind, gamma5, oracle):
    gpu, orc = make(setup, kind, gamma5, oracle)
    x = synth.gaussian_spinor(setup["dims"], 3, 8)
    y = synth.gaussian_spinor(setup["dims"], 3, 9)
    alpha = 0.37 - 0.21j
    out = gpu.multiplyAdd(setup["lat"].new_vector(), x, y, alpha)
    assert rel(out, orc.multiply_add(x, y, alpha)) < 1e-13
    # multiplyAdd(alpha = 0) == multiply (tests/TestLinearAlgebra.cpp:141-144)
    out0 = gpu.multiplyAdd(setup["lat"].new_vector(), x, y, 0.0)
    assert rel(out0, gpu.multiply(x)) < 1e-15


def test_even_odd_multiply_add_unsupported(setup, oracle):
    gpu, _ = make(setup, "EvenOddImproved", True, oracle)
    x = synth.gaussian_spinor(setup["dims"], 3, 10)
    with pytest.raises(L.LymError):
        gpu.multiplyAdd(setup["lat"].new_vector(), x, x, 1.0)


def test_field_strength_matches_oracle(setup, oracle):
    gpu, orc = make(setup, "Improved", True, oracle)
    F = gpu.field_strength()
    Fo = orc.field_strength()
    assert F.shape == Fo.shape
    assert np.abs(F - Fo).max() < 1e-14


def test_gamma5_hermiticity(setup, oracle):
    # TestLinearAlgebra.cpp:36-57: |<y, Q x> - <Q y, x>|^2
    for kind in ("DiracWilson", "Improved"):
        gpu, _ = make(setup, kind, True, oracle)
        x = synth.gaussian_spinor(setup["dims"], 3, 11)
        y = synth.gaussian_spinor(setup["dims"], 3, 12)
        h = np.vdot(y, gpu.multiply(x)) - np.vdot(gpu.multiply(y), x)
        assert abs(h) < 1e-11 * np.linalg.norm(x) * np.linalg.norm(y)


def test_csw_zero_equals_wilson(setup, oracle):
    # TestLinearAlgebra.cpp:122-140
    lat = setup["lat"]
    w = L.DiracWilsonOperator(lat, setup["kappa"])
    w.setLattice(setup["gid"])
    c = L.ImprovedDiracWilsonOperator(lat, setup["kappa"], 0.0)
    c.setLattice(setup["gid"])
    x = synth.gaussian_spinor(setup["dims"], 3, 13)
    assert rel(w.multiply(x), c.multiply(x)) < 1e-15
    assert rel(w.multiplyAdd(x, x, 0.0), c.multiplyAdd(x, x, 0.0)) < 1e-15


@pytest.mark.parametrize("precision,tol", [("single", 1e-6), ("half", 1e-2)])
@pytest.mark.parametrize("kind", ["Improved", "EvenOddImproved", "SquareImproved"])
def test_sloppy_precision_stencil(setup, precision, tol, kind, oracle):
    gpu, orc = make(setup, kind, True, oracle)
    x = synth.gaussian_spinor(setup["dims"], 3, 14)
    assert rel(gpu.multiply_precision(x, precision), orc.multiply(x)) < tol


@pytest.mark.parametrize("kind", ["DiracWilson", "Improved", "EvenOddImproved", "SquareImproved"])
@pytest.mark.parametrize("gamma5", [True, False])
def test_eight_real_links_stencil(setup, kind, gamma5, oracle):
    """The FP32 stencil on SU(3) links stored in 8 reals (lym_set_link_format) against the FP64
    oracle, 1e-6 as the 12-real format; SU(2) adjoint links refuse the format."""
    lat = setup["lat"]
    if setup["rep"] != "su3":
        with pytest.raises(L.LymError):
            lat.set_link_format(8)
        return
    gpu, orc = make(setup, kind, gamma5, oracle)
    x = synth.gaussian_spinor(setup["dims"], 3, 15)
    want = orc.multiply(x)
    try:
        lat.set_link_format(8)
        e8 = rel(gpu.multiply_precision(x, "single"), want)
    finally:
        lat.set_link_format(12)
    e12 = rel(gpu.multiply_precision(x, "single"), want)
    print(f"{kind} gamma5={gamma5}: FP32 stencil error 8 reals {e8:.2e}, 12 reals {e12:.2e}")
    assert e8 < 1e-6 and e12 < 1e-6


def test_eight_real_links_mixed_solve(setup, oracle):
    """The mixed-precision even-odd CG with its FP32 inner iterations on 8-real links still
    reaches the FP64 true residual 1e-10 (re-measured with the oracle)."""
    if setup["rep"] != "su3":
        return
    lat = setup["lat"]
    gpu, orc = make(setup, "Improved", False, oracle)
    b = synth.gaussian_spinor(setup["dims"], 3, 16)
    x = lat.new_vector()
    try:
        lat.set_link_format(8)
        assert L.EvenOddConjugateGradient("single", 1e-10).solve(gpu, b, x)
    finally:
        lat.set_link_format(12)
    assert np.linalg.norm(b - orc.multiply(x)) / np.linalg.norm(b) <= 1e-10


def test_neighbour_tables_bit_exact(setup, oracle):
    sup, sdn = setup["lat"].neighbour_tables()
    osup, osdn, _ = oracle.geom_tables(setup["dims"])
    assert np.array_equal(sup, osup) and np.array_equal(sdn, osdn)


def test_stencil_indices_match_reference_tables(setup, oracle):
    idx = setup["lat"].stencil_indices()
    osup, osdn, coord = oracle.geom_tables(setup["dims"])
    Vh = idx.shape[1]
    for p in range(2):
        lex = idx[p, :, 0]
        assert np.array_equal(lex >> 1, np.arange(Vh))
        assert np.all(coord[lex].sum(axis=1) % 2 == p)
        for mu in range(4):
            assert np.array_equal(idx[p, :, 1 + 2 * mu], osup[lex, mu] >> 1)
            assert np.array_equal(idx[p, :, 2 + 2 * mu], osdn[lex, mu] >> 1)


def test_upload_fundamental_matches_host_conversion(setup, oracle):
    lat = setup["lat"]
    dims = setup["dims"]
    if setup["rep"] == "su3":
        fund = synth.su3_links(dims, 0.3, 99)
        host = synth.antiperiodic_bc(fund, dims)
    else:
        fund = synth.su2_links(dims, 0.3, 99)
        host = synth.antiperiodic_bc(synth.su2_to_adjoint(fund), dims)
    g1 = lat.upload_fundamental(fund, "fermion_antiperiodic")
    g2 = lat.upload(host)
    a = L.ImprovedDiracWilsonOperator(lat, 0.12, 1.1)
    a.setLattice(g1)
    b = L.ImprovedDiracWilsonOperator(lat, 0.12, 1.1)
    b.setLattice(g2)
    x = synth.gaussian_spinor(dims, 3, 15)
    assert rel(a.multiply(x), b.multiply(x)) < 1e-14


@pytest.mark.parametrize("rep", ["su3", "su2adj"])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 4, 2, 6), (4, 2, 6, 4), (2, 2, 4, 10)])
@pytest.mark.parametrize("csw", [1.3, 9.0])
def test_gauge_and_clover_tiles(rep, dims, csw, oracle):
    """Link formats and clover blocks built in tiles of 32 sites: lattices smaller than a tile,
    ragged last tiles, extents of 2; a c_sw so large that T is indefinite and its inverse needs
    the pivoting.  The Schur operator reads T and T^-1 in every precision."""
    kappa = 0.2
    links = synth.fermion_links(dims, rep, 0.6, 29)
    lat = L.Lattice(dims, rep)
    try:
        op = L.EvenOddImprovedDiracWilsonOperator(lat, kappa, csw, gamma5=True)
        op.setLattice(lat.upload(links))
        orc = oracle.Operator(oracle.Geometry(dims), links, "EvenOddImproved", kappa, csw, True)
        F = op.field_strength()
        Fo = orc.field_strength()
        assert np.max(np.abs(F - np.asarray(Fo).reshape(F.shape))) < 1e-14
        x = synth.gaussian_spinor(dims, 3, 31)
        ref = orc.multiply(x)
        # the worst condition number of the even blocks bounds the inverse's rounding
        e = np.eye(12).reshape(12, 4, 3)
        cols = [orc.even_even_inverse(np.broadcast_to(v, (lat.V, 4, 3)).astype(np.complex128).copy()) for v in e]
        Ti = np.stack([c.reshape(lat.V, 12) for c in cols], axis=-1)
        even = np.add.reduce(synth.lex_coords(dims), axis=1) % 2 == 0
        cond = np.linalg.cond(Ti[even]).max()
        assert rel(op.multiply(x), ref) < 1e-14 * cond + 1e-14
        if cond < 1e3:  # the odd sites: the even ones are copied
            assert rel(op.multiply_precision(x, "single")[~even], ref[~even]) < 1e-6 * cond
            assert rel(op.multiply_precision(x, "half")[~even], ref[~even]) < 5e-3 * cond
    finally:
        lat.close()


@pytest.mark.parametrize("rep", ["su3", "su2adj"])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 6, 2, 10), (4, 2, 6, 6), (2, 2, 2, 34)])
@pytest.mark.parametrize("kind", KINDS)
def test_fp64_stencil_tiles(rep, dims, kind, oracle):
    """The FP64 stencil's tiles of 16 and 32 half-sites: fewer half-sites than a tile, ragged last
    tiles, extents of 2; results written straight into device vectors, also over an input."""
    import ctypes as C

    import torch
    kappa, csw = 0.15, 1.1
    links = synth.fermion_links(dims, rep, 0.4, 41)
    lat = L.Lattice(dims, rep)
    try:
        op = GPU_CLASS[kind](lat)
        op.setKappa(kappa)
        if "Wilson" not in kind:
            op.setCSW(csw)
        op.setLattice(lat.upload(links))
        orc = oracle.Operator(oracle.Geometry(dims), links, kind, kappa, 0.0 if "Wilson" in kind else csw, True)
        x, y = (synth.gaussian_spinor(dims, 3, 43 + k) for k in range(2))
        ref, alpha = orc.multiply(x), 0.3 - 0.2j
        assert rel(op.multiply(x), ref) < 1e-13

        def call(name, out, *args):
            torch.cuda.synchronize()
            rc = getattr(L.lib(), name)(lat.handle, op.op_id, *[C.c_void_p(v.data_ptr()) for v in (out, *args[:2])],
                                        *args[2:])
            assert rc == 0
            return out.cpu().numpy()

        dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        assert rel(call("lym_multiply_device", dx, dx), ref) < 1e-13  # over its input
        if kind == "EvenOddImproved":
            return
        refa, a = ref + alpha * y, (alpha.real, alpha.imag)
        for case in ("apart", "over v2", "over v1"):
            dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
            out = {"apart": torch.empty_like(dx), "over v2": dy, "over v1": dx}[case]
            assert rel(call("lym_multiply_add_device", out, dx, dy, *a), refa) < 1e-13
        # v2 and the result overlap in part
        buf = torch.zeros((lat.V + 1, 4, 3), dtype=torch.complex128, device="cuda")
        buf[1:] = torch.from_numpy(y).cuda()
        dx = torch.from_numpy(x).cuda()
        assert rel(call("lym_multiply_add_device", buf[:-1], dx, buf[1:], *a), refa) < 1e-13
    finally:
        lat.close()


@pytest.mark.parametrize("dims", [(8, 8, 8, 24), (8, 8, 8, 26)])
@pytest.mark.parametrize("kind,rep", [("DiracWilson", "su3"), ("Improved", "su3"), ("Improved", "su2adj")])
def test_input_read_in_place_or_packed(kind, rep, dims, oracle):
    """Either side of the size up to which an application reads the caller's vector in the stencil
    itself; a result over the input is packed first on both."""
    import ctypes as C

    import torch
    kappa, csw = 0.13, 1.0
    links = synth.fermion_links(dims, rep, 0.4, 47)
    lat = L.Lattice(dims, rep)
    try:
        op = GPU_CLASS[kind](lat)
        op.setKappa(kappa)
        if kind != "DiracWilson":
            op.setCSW(csw)
        op.setLattice(lat.upload(links))
        orc = oracle.Operator(oracle.Geometry(dims), links, kind, kappa, 0.0 if kind == "DiracWilson" else csw, True)
        x = synth.gaussian_spinor(dims, 3, 48)
        ref = orc.multiply(x)
        for over in (False, True):
            dx = torch.from_numpy(x).cuda()
            out = dx if over else torch.empty_like(dx)
            torch.cuda.synchronize()
            assert L.lib().lym_multiply_device(lat.handle, op.op_id, C.c_void_p(out.data_ptr()),
                                               C.c_void_p(dx.data_ptr())) == 0
            assert rel(out.cpu().numpy(), ref) < 1e-13
    finally:
        lat.close()


@pytest.mark.parametrize("dims", [(3, 2, 4, 6), (4, 5, 2, 4), (2, 2, 3, 10), (3, 5, 7, 2), (4, 2, 6, 4)])
@pytest.mark.parametrize("kind", ["DiracWilson", "Improved", "SquareImproved"])
def test_odd_extents_are_one_operator(kind, dims):
    """With odd space extents too every way of applying an operator gives the same vector: apart,
    over the input (packed first), with an added vector that overlaps the result (the general
    path), and twice for the square."""
    import ctypes as C

    import torch
    links = synth.fermion_links(dims, "su3", 0.4, 51)
    lat = L.Lattice(dims, "su3")
    try:
        gid = lat.upload(links)

        def make(kind):
            op = GPU_CLASS[kind](lat)
            op.setKappa(0.14)
            if kind != "DiracWilson":
                op.setCSW(1.1)
            op.setLattice(gid)
            return op

        op = make(kind)
        x = synth.gaussian_spinor(dims, 3, 52)

        def call(op, out, v, add=None):
            torch.cuda.synchronize()
            p = [C.c_void_p(t.data_ptr()) for t in (out, v)]
            if add is None:
                rc = L.lib().lym_multiply_device(lat.handle, op.op_id, *p)
            else:
                rc = L.lib().lym_multiply_add_device(lat.handle, op.op_id, *p, C.c_void_p(add.data_ptr()), 0.0, 0.0)
            assert rc == 0
            return out.cpu().numpy()

        dx = torch.from_numpy(x).cuda()
        apart = call(op, torch.empty_like(dx), dx)
        over = torch.from_numpy(x).cuda()
        buf = torch.zeros((lat.V + 1, 4, 3), dtype=torch.complex128, device="cuda")
        assert rel(call(op, over, over), apart) < 1e-14
        assert rel(call(op, buf[:-1], dx, buf[1:]), apart) < 1e-14
        if kind == "SquareImproved":
            d = make("Improved")
            once = call(d, torch.empty_like(dx), dx)
            assert rel(call(d, torch.empty_like(dx), torch.from_numpy(once).cuda()), apart) < 1e-13
    finally:
        lat.close()
