"""Measured cases of the library: what a lattice program has it do, through the C ABI.

Every case holds what such a program holds before the call (a lattice context with resident
links, an operator, source and result buffers in device memory) and one pass is one call of
the public entry points: an operator application, a solve, a block solve, a multishift solve,
a fermion force, a new gauge field with its first application, meson contractions.

Links are smooth SU(3) (or adjoint SU(2)) matrices, antiperiodic in time; vectors are complex
normal.  Every extent is even (the even-odd split), powers of two and others alike.  exact()
restates the same quantities in plain torch, complex128, on full-lattice arrays.
"""
import ctypes as C
import math

import numpy as np
import torch

import leonardym_b200 as L
from leonardym_b200 import solvers
from leonardym_b200._lib import SolveStats, lib

DEV = "cuda"
TOL = 1e-10  # relative residual of every solve

SOLVERS = {"cg": solvers.SOLVER_CG, "eo_cg_double": solvers.SOLVER_EO_CG,
           "eo_cg_single": solvers.SOLVER_EO_CG_MIXED_SINGLE, "eo_cg_half": solvers.SOLVER_EO_CG_MIXED_HALF,
           "eo_bicgstab_single": solvers.SOLVER_EO_BICGSTAB_MIXED_SINGLE,
           "eo_bicgstab_half": solvers.SOLVER_EO_BICGSTAB_MIXED_HALF}
OPERATORS = {"Improved": L.ImprovedDiracWilsonOperator, "EvenOddImproved": L.EvenOddImprovedDiracWilsonOperator,
             "SquareImproved": L.SquareImprovedDiracWilsonOperator,
             "SquareEvenOddImproved": L.SquareEvenOddImprovedDiracWilsonOperator}


def _case(path, dims, rep="su3", **more):
    kappa, csw = (0.137, 1.7) if rep == "su3" else (0.175, 1.5)
    case = {"path": path, "rep": rep, "x": dims[0], "y": dims[1], "z": dims[2], "t": dims[3], "kappa": kappa,
            "csw": csw}
    case.update(more)
    return case


def listed():
    return [
        # one application of the Wilson-clover operator on the smallest lattice in use: the
        # inner call of a solver that a program drives itself, latency only
        _case("apply", (8, 8, 8, 8), name="apply_8c8", operator="Improved", kappa=0.12, csw=1.0),
        # the same on the lattice of the headline benchmark
        _case("apply", (24, 24, 24, 48), name="apply_24c48", operator="Improved"),
        # the RHMC operator with a shift (multiplyAdd), adjoint SU(2) links
        _case("apply_add", (16, 16, 16, 32), "su2adj", name="apply_add_sq_16c32_adj",
              operator="SquareEvenOddImproved"),
        # CG on D^+ D in double precision, the reference's plain solver, on a small lattice
        _case("solve", (8, 8, 8, 8), name="cg_8c8", operator="SquareImproved", solver="cg", kappa=0.12, csw=1.0),
        # one source, adjoint SU(2): even-odd CG with single-precision inner iterations
        _case("solve", (16, 16, 16, 32), "su2adj", name="eo_cg_single_16c32_adj", operator="Improved",
              solver="eo_cg_single"),
        # the 12 point sources of a meson propagator: block BiCGStab
        _case("block", (24, 24, 24, 48), name="propagator_24c48", operator="Improved", solver="eo_bicgstab_single",
              sources=12, point=True, host=False),
        # noise sources in host memory, half-precision inner storage, a ragged lattice
        _case("block", (14, 10, 12, 22), name="block_half_14x10x12x22_host", operator="Improved",
              solver="eo_bicgstab_half", sources=8, point=False, host=True, kappa=0.13),
        # RHMC: 12 shifts on one pseudofermion with the mixed-precision multishift
        _case("multishift", (24, 24, 24, 48), name="multishift_mixed_24c48", operator="SquareEvenOddImproved",
              algorithm="multishift_cg_mixed_half", shifts=12, kappa=0.1365),
        # the same system in double precision on a ragged lattice
        _case("multishift", (10, 12, 14, 18), name="multishift_fp64_10x12x14x18", operator="SquareEvenOddImproved",
              algorithm="multishift_cg", shifts=8, kappa=0.1365),
        # RHMC: the fermion force of 12 shifts
        _case("force", (24, 24, 24, 48), name="force_24c48", operator="Improved", pairs=12, kappa=0.1365),
        # one molecular-dynamics step's new gauge field: links made resident, clover term built,
        # first application of the even-odd operator
        _case("gauge", (20, 20, 20, 40), name="gauge_20c40", operator="EvenOddImproved"),
        # meson contractions of 12 propagators
        _case("meson", (24, 24, 24, 48), name="meson_24c48"),
    ]


def _even(rng, lo, hi):
    """An even extent, log-uniform in [lo, hi]."""
    return max(lo, min(hi, 2 * round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))) / 2)))


def draw(rng):
    def dims(most):
        while True:
            d = (_even(rng, 4, 28), _even(rng, 4, 28), _even(rng, 4, 28), _even(rng, 6, 64))
            if 2048 <= d[0] * d[1] * d[2] * d[3] <= most:
                return d

    full, mid, small = 24 ** 3 * 48, 16 ** 3 * 32, 12 ** 3 * 24
    path = rng.choice(["apply", "apply", "apply_add", "solve", "solve", "block", "multishift", "force", "gauge",
                       "meson"])
    rep = rng.choice(["su3", "su3", "su2adj"])
    kappa = round(rng.uniform(0.12, 0.135) if rep == "su3" else rng.uniform(0.16, 0.175), 4)
    if path == "apply":
        return _case(path, dims(full), rep, operator=rng.choice(sorted(OPERATORS)), kappa=kappa)
    if path == "apply_add":
        return _case(path, dims(full), rep, operator=rng.choice(["Improved", "SquareEvenOddImproved"]), kappa=kappa)
    if path == "solve":
        solver = rng.choice(["cg", "eo_cg_double", "eo_cg_single", "eo_cg_half"])
        return _case(path, dims(mid if solver != "cg" else small), rep, kappa=kappa, solver=solver,
                     operator="SquareImproved" if solver == "cg" else "Improved")
    if path == "block":
        return _case(path, dims(mid), "su3", operator="Improved", sources=rng.randint(2, 24),
                     solver=rng.choice(["eo_bicgstab_single", "eo_bicgstab_half", "eo_cg_single"]),
                     point=rng.random() < 0.5, host=rng.random() < 0.3, kappa=round(rng.uniform(0.12, 0.135), 4))
    if path == "multishift":
        algorithm = rng.choice(["multishift_cg_mixed_half", "multishift_cg_mixed_single", "multishift_cg"])
        return _case(path, dims(mid if "mixed" in algorithm else small), rep, operator="SquareEvenOddImproved",
                     algorithm=algorithm, shifts=rng.randint(4, 16), kappa=kappa)
    if path == "force":
        return _case(path, dims(full), rep, operator="Improved", pairs=rng.randint(1, 12), kappa=kappa)
    if path == "gauge":
        return _case(path, dims(full), rep, operator=rng.choice(["Improved", "EvenOddImproved"]), kappa=kappa)
    return _case("meson", dims(full), rep, kappa=kappa)


# ------------------------------------------------------------------ inputs --
def _dims(case):
    return case["x"], case["y"], case["z"], case["t"]


def _volume(case):
    return case["x"] * case["y"] * case["z"] * case["t"]


def _links(case, gen):
    """Fermion links [V, 4, 3, 3] in the library's layout ([j, i] = U(i, j)), antiperiodic."""
    V, eps = _volume(case), 0.25
    if case["rep"] == "su3":
        # rows of 1 + i eps H + (i eps H)^2 / 2, H Hermitian of unit-variance Gell-Mann
        # coefficients, orthonormalised; the third row from the other two
        a = torch.randn((8, 4 * V), generator=gen, device=DEV, dtype=torch.float64)
        H = torch.zeros((4 * V, 3, 3), device=DEV, dtype=torch.complex128)
        d = a[7] / math.sqrt(3.0)
        H[:, 0, 0], H[:, 1, 1], H[:, 2, 2] = a[2] + d, d - a[2], -2 * d
        for k, (i, j) in ((0, (0, 1)), (3, (0, 2)), (5, (1, 2))):
            z = torch.complex(a[k], -a[k + 1])
            H[:, i, j], H[:, j, i] = z, z.conj()
        M = (1j * eps) * H
        U = M + 0.5 * (M @ M)
        U[:, (0, 1, 2), (0, 1, 2)] += 1.0
        r0 = U[:, 0] / U[:, 0].norm(dim=-1, keepdim=True)
        r1 = U[:, 1] - (r0.conj() * U[:, 1]).sum(-1, keepdim=True) * r0
        r1 = r1 / r1.norm(dim=-1, keepdim=True)
        U = torch.stack([r0, r1, torch.linalg.cross(r0, r1).conj()], dim=1)
    else:
        # the rotation of the unit quaternion (cos, sin n) of an SU(2) link
        n = torch.randn((4 * V, 3), generator=gen, device=DEV, dtype=torch.float64)
        th = eps * n.norm(dim=-1, keepdim=True)
        v = n / n.norm(dim=-1, keepdim=True) * th.sin()
        w = th.cos()[:, 0]
        x, y, z = v[:, 0], v[:, 1], v[:, 2]
        U = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y),
                         2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x),
                         2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], dim=1).view(-1, 3, 3)
    links = U.transpose(-1, -2).contiguous().view(V, 4, 3, 3)
    links.view(-1, case["t"], 4, 3, 3)[:, -1, 3] *= -1
    return links


def _vector(case, gen):
    a = torch.randn((_volume(case), 4, 3, 2), generator=gen, device=DEV, dtype=torch.float64) * math.sqrt(0.5)
    return torch.view_as_complex(a)


def _inputs(case, seed):
    """Links and the call's vectors, on the device, from the seed alone."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    inp = {"links": _links(case, gen) if case["path"] != "meson" else None}
    path = case["path"]
    if path == "apply_add":
        inp["vectors"] = [_vector(case, gen) for _ in range(2)]
    elif path == "force":
        inp["vectors"] = [_vector(case, gen) for _ in range(2 * case["pairs"])]
        inp["weights"] = [0.5 / (1.0 + k) for k in range(case["pairs"])]
    elif path == "meson":
        # a propagator falls off with the distance in time from its source
        t = torch.arange(case["t"], device=DEV, dtype=torch.float64)
        fall = torch.exp(-0.4 * torch.minimum(t, case["t"] - t)).view(1, -1, 1, 1)
        inp["vectors"] = [(_vector(case, gen).view(-1, case["t"], 4, 3) * fall).view(-1, 4, 3) for _ in range(12)]
    elif path == "block" and case["point"]:
        vs = []
        for k in range(case["sources"]):
            v = torch.zeros((_volume(case), 4, 3), device=DEV, dtype=torch.complex128)
            v[(k // 12) * 2, k % 4, (k // 4) % 3] = 1.0
            vs.append(v)
        inp["vectors"] = vs
    elif path == "block":
        # Z2 x Z2 noise
        vs = []
        for _ in range(case["sources"]):
            b = torch.randint(0, 2, (_volume(case), 4, 3, 2), generator=gen, device=DEV).to(torch.float64)
            vs.append(torch.view_as_complex((2 * b - 1) * math.sqrt(0.5)))
        inp["vectors"] = vs
    else:
        inp["vectors"] = [_vector(case, gen)]
    return inp


def _shifts(case):
    n = case["shifts"]
    return [10.0 ** (-4 + 4.0 * k / (n - 1)) for k in range(n)]


def _pointers(tensors):
    return (C.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])


def _p(tensor):
    return C.c_void_p(tensor.data_ptr())


def prepare(case, seed):
    inp = _inputs(case, seed)
    path = case["path"]
    st = {"case": case, "vectors": inp["vectors"]}
    lat = st["lattice"] = L.Lattice(_dims(case), case["rep"])
    st["ctx"] = lat.handle
    if inp["links"] is not None:
        torch.cuda.synchronize()  # the library's stream does not wait for torch's
        _check(st, lib().lym_gauge_upload_device(st["ctx"], 1, _p(inp["links"])))
        # D x = b is solved without gamma5, everything else runs the Hermitian operator
        op = OPERATORS[case["operator"]](lat, case["kappa"], case["csw"],
                                         gamma5=path not in ("block", "force") and case.get("solver") in (None, "cg"))
        op.setLattice(1)
        st["op"], st["op_id"] = op, op.op_id
    if path == "gauge":
        st["links"] = inp["links"]
    vs = inp["vectors"]
    if path in ("apply", "apply_add", "gauge", "solve"):
        st["out"] = torch.zeros_like(vs[0])
    elif path == "block":
        if case["host"]:
            st["vectors"] = vs = [v.cpu().pin_memory() for v in vs]
            st["out"] = [torch.zeros(v.shape, dtype=v.dtype, pin_memory=True) for v in vs]
        else:
            st["out"] = [torch.zeros_like(v) for v in vs]
        st["sources"], st["solutions"] = _pointers(vs), _pointers(st["out"])
        st["stats"] = (SolveStats * len(vs))()
    elif path == "multishift":
        st["out"] = [torch.zeros_like(vs[0]) for _ in range(case["shifts"])]
        st["solutions"] = _pointers(st["out"])
        st["shifts"] = np.array(_shifts(case))
        st["stats"] = SolveStats()
        st["precision"] = TOL ** 2 * float(vs[0].abs().square().sum())
    elif path == "force":
        n = case["pairs"]
        st["X"], st["Y"] = _pointers(vs[:n]), _pointers(vs[n:])
        st["weights"] = np.array(inp["weights"])
        st["out"] = torch.zeros((_volume(case), 4, 3, 3), dtype=torch.complex128, device=DEV)
    elif path == "meson":
        st["props"] = _pointers(vs)
        st["out"] = [np.zeros(case["t"]) for _ in range(3)]
    if path == "solve":
        st["stats"] = SolveStats()
        # CG takes the reference's absolute threshold on the squared residual, the even-odd
        # solvers a relative tolerance
        st["precision"] = TOL ** 2 * float(vs[0].abs().square().sum()) if case["solver"] == "cg" else -TOL
    torch.cuda.synchronize()
    return st


def _check(st, rc):
    if rc != 0:
        raise L.LymError(rc, (lib().lym_last_error(st["ctx"]) or b"").decode())


def run(st):
    case, ctx, api = st["case"], st["ctx"], lib()
    path, out, vs = case["path"], st["out"], st["vectors"]
    if path == "apply":
        _check(st, api.lym_multiply_device(ctx, st["op_id"], _p(out), _p(vs[0])))
    elif path == "apply_add":
        _check(st, api.lym_multiply_add_device(ctx, st["op_id"], _p(out), _p(vs[0]), _p(vs[1]), 0.01, 0.0))
    elif path == "gauge":
        _check(st, api.lym_gauge_upload_device(ctx, 1, _p(st["links"])))
        _check(st, api.lym_multiply_device(ctx, st["op_id"], _p(out), _p(vs[0])))
    elif path == "solve":
        _check(st, api.lym_solve_device(ctx, st["op_id"], SOLVERS[case["solver"]], st["precision"], 20000, _p(vs[0]),
                                        _p(out), None, C.byref(st["stats"])))
    elif path == "block":
        solve = api.lym_solve_block if case["host"] else api.lym_solve_block_device
        _check(st, solve(ctx, st["op_id"], SOLVERS[case["solver"]], -TOL, 20000, len(vs), st["sources"],
                         st["solutions"], 16, st["stats"]))
    elif path == "multishift":
        _check(st, api.lym_multishift_device(ctx, st["op_id"], solvers.MULTISHIFT[case["algorithm"]], case["shifts"],
                                             st["shifts"].ctypes.data_as(C.c_void_p), st["precision"], 20000,
                                             _p(vs[0]), st["solutions"], C.byref(st["stats"])))
    elif path == "force":
        out.zero_()
        torch.cuda.current_stream().synchronize()  # the library's stream does not wait for torch's
        _check(st, api.lym_fermion_force_multi_device(ctx, st["op_id"], case["pairs"], st["X"], st["Y"],
                                                      st["weights"].ctypes.data_as(C.c_void_p), _p(out)))
    else:
        _check(st, api.lym_meson_contractions_device(ctx, st["props"], *[o.ctypes.data_as(C.c_void_p) for o in out]))
    return out


# -------------------------------------------------------------------- work --
# operator applications (of S, or of D for plain CG) of a solve to 1e-10 at these couplings
_APPLICATIONS = {"cg": 2 * 106, "eo_cg_double": 2 * 105, "eo_cg_single": 2 * 109, "eo_cg_half": 2 * 115,
                 "eo_bicgstab_single": 2 * 90, "eo_bicgstab_half": 2 * 36}


def work(case):
    V = _volume(case)
    word = 8.0
    link, hop = (18, 1320) if case["rep"] == "su3" else (9, 768)
    vec = 24.0 * V * word
    field = (4 * link + 72.0) * V  # link and clover reals
    flops = (hop + 504 + 48.0) * V  # one application of D or of S
    path = case["path"]
    if path in ("apply", "apply_add"):
        twice = 2 if case["operator"].startswith("Square") else 1
        return {"bytes": field * word + (2 if path == "apply" else 3) * vec, "flops": twice * flops}
    if path == "gauge":
        # links in, operator's vectors; per site 6 planes of 4 leaves of 3 matrix products and
        # two 6 x 6 inverses
        return {"bytes": 4 * link * V * word + 2 * vec, "flops": V * (24 * 3 * 198 + 2 * 1700.0) + flops}
    if path == "force":
        # per link and plane 16 matrix products, per pair the outer products
        n = case["pairs"]
        return {"bytes": 2 * n * vec + (4 * link + 2 * 72.0) * V * word,
                "flops": V * (12 * 16 * 198.0 + n * (6 * 8 * 72.0 + 4 * 8 * 150.0))}
    if path == "meson":
        return {"bytes": 12 * vec, "flops": V * 144 * 20.0}
    if path == "multishift":
        n, mixed = case["shifts"], "mixed" in case["algorithm"]
        its = 280 if mixed else 186
        word = 4.0 if mixed else 8.0
        # an iteration: two applications of S and the base system's three vectors
        return {"bytes": its * (2 * field + 6 * 12.0 * V) * word + (n + 1) * vec, "flops": its * 2 * flops}
    n = case.get("sources", 1)
    word = 8.0 if case["solver"] in ("cg", "eo_cg_double") else 4.0 if "single" in case["solver"] else 2.0
    a = _APPLICATIONS[case["solver"]]
    # every application reads the fields once for a batch of 16 and moves each source's vectors
    return {"bytes": a * (math.ceil(n / 16) * field + n * 3 * 12.0 * V) * word + 2 * n * vec, "flops": n * a * flops}


def tolerance(case):
    path = case["path"]
    # double-precision sums: 1.5e-16 to 6e-16 off exact(); meson sums cancel, up to 1e-15
    if path in ("apply", "apply_add", "gauge", "force"):
        return {"rel": 4e-15, "max": 4e-14}
    if path == "meson":
        return {"rel": 1e-14, "max": 1e-13}
    # solutions to a relative residual of 1e-10, times the condition of the operator: up to
    # 2e-9 off exact() at the smallest shift, and as much between two stopping points
    return {"rel": 1.2e-8, "max": 5e-7}


# ------------------------------------------------------------------- exact --
_PARTNER = ((3, 2), (3, 2), (2, 3), (2, 3))
_CODE = ((-1j, -1j), (-1.0, 1.0), (-1j, 1j), (1.0, 1.0))


class _Exact:
    """Wilson-clover operators on [x, y, z, t, 4, 3] arrays in complex128."""

    def __init__(self, case, links, clover=True):
        self.case, self.dims = case, _dims(case)
        lk = links.to(torch.complex128).view(*self.dims, 4, 3, 3)
        self.lt = [lk[..., mu, :, :].contiguous() for mu in range(4)]  # U_mu transposed
        self.kappa = case["kappa"]
        n = sum(torch.arange(d, device=DEV).view([-1 if k == m else 1 for k in range(4)])
                for m, d in enumerate(self.dims))
        self.odd = (n % 2).to(torch.float64).view(*self.dims, 1, 1)
        self.even = 1.0 - self.odd
        self.code = [torch.tensor(c, device=DEV, dtype=torch.complex128).view(2, 1) for c in _CODE]
        if clover:
            self.T = self._clover()
            self.Ti = torch.linalg.inv(self.T)

    def u(self, mu):
        return self.lt[mu].transpose(-1, -2)

    def shape(self, v):
        return v.reshape(*self.dims, 4, 3)

    def _clover(self):
        def at(m, mu=None, by=0, nu=None, by2=0):
            m = torch.roll(m, -by, mu) if by else m
            return torch.roll(m, -by2, nu) if by2 else m

        def dag(m):
            return m.conj().transpose(-1, -2)

        F = []
        for mu, nu in ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)):
            um, un = self.u(mu), self.u(nu)
            # the plaquette leaf in the positive quadrant, and the other three
            P = um @ at(un, mu, 1) @ dag(at(um, nu, 1)) @ dag(un)
            Q = P
            Q = Q + un @ dag(at(um, mu, -1, nu, 1)) @ dag(at(un, mu, -1)) @ at(um, mu, -1)
            Q = Q + dag(at(um, mu, -1)) @ dag(at(un, mu, -1, nu, -1)) @ at(um, mu, -1, nu, -1) @ at(un, nu, -1)
            Q = Q + dag(at(un, nu, -1)) @ at(um, nu, -1) @ at(un, mu, 1, nu, -1) @ dag(um)
            F.append(0.125 * (Q - dag(Q)))
        kc = self.case["kappa"] * self.case["csw"]
        T = torch.zeros((*self.dims, 2, 6, 6), device=DEV, dtype=torch.complex128)
        T[..., 0, :3, :3], T[..., 0, 3:, 3:] = 1j * (F[5] - F[0]), 1j * (F[0] - F[5])
        T[..., 0, :3, 3:], T[..., 0, 3:, :3] = F[1] + F[4] + 1j * (F[2] - F[3]), -F[1] - F[4] + 1j * (F[2] - F[3])
        T[..., 1, :3, :3], T[..., 1, 3:, 3:] = -1j * (F[0] + F[5]), 1j * (F[0] + F[5])
        T[..., 1, :3, 3:], T[..., 1, 3:, :3] = F[1] - F[4] - 1j * (F[2] + F[3]), F[4] - F[1] - 1j * (F[2] + F[3])
        T *= kc
        T += torch.eye(6, device=DEV, dtype=torch.complex128)
        return T

    def block(self, M, x):
        return (M @ x.reshape(*self.dims, 2, 6, 1)).view(*self.dims, 4, 3)

    def hop(self, x):
        """sum over mu of U (1 - gamma) x(s + mu) + U^+ (1 + gamma) x(s - mu)."""
        out = torch.zeros_like(x)
        for mu in range(4):
            p, c = list(_PARTNER[mu]), self.code[mu]
            up, low = x[..., :2, :], c * x[..., p, :]
            w = torch.roll(up - low, -1, mu) @ self.lt[mu]
            out[..., :2, :] += w
            out[..., p, :] -= c.conj() * w
            w = torch.roll((up + low) @ self.lt[mu].conj().transpose(-1, -2), 1, mu)
            out[..., :2, :] += w
            out[..., p, :] += c.conj() * w
        return out

    @staticmethod
    def gamma5(x):
        return torch.cat([x[..., :2, :], -x[..., 2:, :]], dim=-2)

    def D(self, x):
        return self.block(self.T, x) - self.kappa * self.hop(x)

    def S(self, x):  # odd sites in and out
        e = self.even * self.block(self.Ti, self.even * self.hop(x))
        return self.odd * (self.block(self.T, x) - self.kappa ** 2 * self.hop(e))

    def Q(self, x):
        return self.gamma5(self.S(x))

    def apply(self, x):
        name = self.case["operator"]
        if name == "Improved":
            return self.gamma5(self.D(x))
        if name == "SquareImproved":
            return self.gamma5(self.D(self.gamma5(self.D(x))))
        o = self.Q(self.odd * x)
        return self.even * x + (self.Q(o) if name.startswith("Square") else o)

    @staticmethod
    def cg(A, b, rel):
        x = torch.zeros_like(b)
        r, p = b.clone(), b.clone()
        rr = torch.vdot(r.flatten(), r.flatten()).real
        stop = rel * rel * float(rr)
        for it in range(20000):
            if it % 8 == 0 and float(rr) <= stop:
                break
            ap = A(p)
            a = rr / torch.vdot(p.flatten(), ap.flatten()).real
            x += a * p
            r -= a * ap
            new = torch.vdot(r.flatten(), r.flatten()).real
            p = r + (new / rr) * p
            rr = new
        return x

    def solve(self, b, rel=1e-13):
        """D x = b through the odd sites."""
        be, bo = self.even * b, self.odd * b
        bo = bo + self.kappa * self.odd * self.hop(self.even * self.block(self.Ti, be))
        x = self.cg(lambda v: self.Q(self.Q(v)), self.Q(self.gamma5(bo)), rel)
        return x + self.even * self.block(self.Ti, be + self.kappa * self.even * self.hop(x))

    def force(self, X, Y, weights):
        """sum_i w_i F(X_i, Y_i) as [x, y, z, t, 4, 3, 3] matrices."""
        eye = torch.eye(4, device=DEV, dtype=torch.complex128)
        g5 = torch.diag(torch.tensor([1, 1, -1, -1], device=DEV, dtype=torch.complex128))
        gam = []
        for mu in range(4):
            g = torch.zeros((4, 4), device=DEV, dtype=torch.complex128)
            for k in range(2):
                g[k, _PARTNER[mu][k]] = _CODE[mu][k]
                g[_PARTNER[mu][k], k] = complex(_CODE[mu][k]).conjugate()
            gam.append(g)
        kappa, kc = self.kappa, self.kappa * self.case["csw"]
        X, Y = [self.shape(v) for v in X], [self.shape(v) for v in Y]

        def dag(m):
            return m.conj().transpose(-1, -2)

        def spin(G, v):
            return torch.einsum("ab,...bi->...ai", G, v)

        def outer(y, x):  # sum over spin of y_i conj(x_j)
            return y.transpose(-1, -2) @ x.conj()

        F = torch.zeros((*self.dims, 4, 3, 3), device=DEV, dtype=torch.complex128)
        for mu in range(4):
            U, mg, pg = self.u(mu), g5 @ (eye - gam[mu]), g5 @ (eye + gam[mu])
            for x, y, w in zip(X, Y, weights):
                for a, b in ((x, y), (y, x)):
                    af, bf = torch.roll(a, -1, mu), torch.roll(b, -1, mu)
                    F[..., mu, :, :] -= kappa * w * outer(spin(mg, bf), a)
                    # U^+ b and U a(x + mu), rows of colour
                    F[..., mu, :, :] += kappa * w * outer(spin(pg, b) @ U.conj(), af @ self.lt[mu])
        for mu in range(4):
            for nu in range(4):
                if mu == nu:
                    continue
                sig = g5 @ (0.5j * (gam[mu] @ gam[nu] - gam[nu] @ gam[mu]))
                N = 0
                for x, y, w in zip(X, Y, weights):
                    # N_ij = sum_ab sig_ab (y_b,i conj(x_a,j) + x_b,i conj(y_a,j))
                    N = N + (1j * kc * w) * (outer(spin(sig, y), x) + outer(spin(sig, x), y))
                um, un = self.u(mu), self.u(nu)
                f = lambda m, *d: torch.roll(m, [-k for k in d[1::2]], list(d[0::2]))  # noqa: E731
                un_m, um_n = f(un, mu, 1), f(um, nu, 1)
                A = un_m @ dag(um_n)
                t = A @ f(N, nu, 1) @ dag(un) + A @ dag(un) @ N
                D = un @ um_n
                t = t + un_m @ f(N, mu, 1, nu, 1) @ dag(D) + f(N, mu, 1) @ un_m @ dag(D)
                um_b, un_b, un_mb = f(um, nu, -1), f(un, nu, -1), f(un, mu, 1, nu, -1)
                Cm, R = dag(um) @ dag(un_b), um @ dag(un_mb)
                Lm, B = Cm @ um_b, um @ dag(un_mb) @ dag(um_b)
                t = t - Lm @ f(N, mu, 1, nu, -1) @ dag(R) - Lm @ un_mb @ f(N, mu, 1) @ dag(um)
                t = t - Cm @ f(N, nu, -1) @ dag(B) - dag(um) @ N @ dag(B @ un_b)
                F[..., mu, :, :] += 0.25 * t
        return F


def exact(case, seed):
    inp = _inputs(case, seed)
    vs, path = inp["vectors"], case["path"]
    if path == "meson":
        S = torch.stack(vs).view(3, 4, -1, case["t"], 4, 3)  # source colour, source spin, space, t, spin, colour
        sign = torch.tensor([1.0, 1.0, -1.0, -1.0], device=DEV, dtype=torch.float64)
        perm = [2, 3, 0, 1]
        out = [torch.zeros(case["t"], device=DEV, dtype=torch.float64) for _ in range(3)]
        for c in range(3):
            G = S[c]
            out[0] += G.abs().square().sum((0, 1, 3, 4))
            H = G[perm][:, :, :, perm]
            out[1] += ((G.conj() * H).real.sum((1, 4)) * sign.view(-1, 1, 1) * sign).sum((0, 2))
            out[2] += (G.conj() * G[:, :, :, perm]).real.sum((0, 1, 3, 4))
            out[2] -= (G.conj() * G[perm]).real.sum((0, 1, 3, 4))
        return out
    E = _Exact(case, inp["links"], clover=path != "force")
    if path in ("apply", "gauge", "apply_add"):
        y = E.apply(E.shape(vs[0]))
        return (y + 0.01 * E.shape(vs[1]) if path == "apply_add" else y).reshape(-1, 4, 3)
    if path == "force":
        n = case["pairs"]
        F = E.force(vs[:n], vs[n:], inp["weights"])
        return -F.transpose(-1, -2).reshape(-1, 4, 3, 3).contiguous()
    if path == "solve":
        b = E.shape(vs[0])
        x = E.cg(E.apply, b, 1e-13) if case["solver"] == "cg" else E.solve(b)
        return x.reshape(-1, 4, 3)
    if path == "block":  # the first source
        return [E.solve(E.shape(vs[0])).reshape(-1, 4, 3)] + [None] * (len(vs) - 1)
    # multishift: the smallest and the largest shift
    b, out = E.shape(vs[0]), [None] * case["shifts"]
    for k in (0, case["shifts"] - 1):
        s = _shifts(case)[k]
        x = E.cg(lambda v: E.Q(E.Q(v)) + s * v, E.odd * b, 1e-13)
        out[k] = (x + E.even * b / (1.0 + s)).reshape(-1, 4, 3)
    return out
