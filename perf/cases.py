"""What the engine's speed is measured on: the calls that lattice programs spend their time in.

Every case is one call sequence of a user's program on one lattice (`kind`):

  operator   Hphi_sq on one field: what every observable and solver is made of
  cg         cg_inverter (FP64), the reference's solver, as the HMC monomials call it
  mixed      cg_mixed, the default mixed-precision solve of the same system
  multi      cg_mixed_multi: the point-source propagators of a measurement in one call
  rational   rational_calc: the twelve-pole x^(-1/2) of an RHMC pseudo-fermion
  md_step    one molecular-dynamics step: gauge force, fermion force with the clover
             determinant, the link update and the rebuilt clover term and its inverse
  lattices   cg_inverter_lattices: small lattices of different sizes in one call
  network    the learned preconditioner on one residual (a step of flexible GCR)
  training   its loss and weight gradients over two training pairs

Gauge fields are short Langevin runs of the Wilson action from a cold start at the usual
couplings, so that links have the roughness of a real ensemble; long directions repeat a
smaller field (its extent the smallest even divisor from 8 on), as the benchmark's does.
`exact` evaluates the same quantities in plain torch at 64 bits from their definitions: the
Wilson-clover operator as sums over gamma matrices, forces as derivatives of the action by
autograd, solves by a textbook CG.
"""
import functools
import math

import numpy as np
import torch

from yahmc_b200 import Lattice, Ptc, cg_inverter_lattices

C128 = torch.complex128
DEVICE = "cuda"
TRAINING_PAIRS = 2
DT = 0.05                                    # an outer step of a unit trajectory
C0 = 1.0 + 8.0 / 12.0                        # tree-level Symanzik gauge action
POLES = [46.349181896446986, 9.88019100513198, 3.401308613210369, 1.3630048793095269, 0.5790290064490238,
         0.2514505491704606, 0.10960905737116455, 0.047218180096815734, 0.01961196127354033, 0.007420709380771285,
         0.002168002465687366, 0.000216308812880537]
RESIDUES = [4.567964355025849, 1.2099409193683845, 0.567171139356322, 0.32573707100672644, 0.20375066401778313,
            0.13244732997751965, 0.08782293029116636, 0.05911944846384721, 0.04061338375587007,
            0.028955101338838336, 0.022129375643468088, 0.01898070388006642]
A0 = 0.045504119038756896                    # x^(-1/2) on [0.0052, 8]


def _case(kind, dims, nc=3, repr="fundamental", mass=-0.6, **more):
    t, x, y, z = dims
    return {"kind": kind, "t": t, "x": x, "y": y, "z": z, "nc": nc, "repr": repr, "mass": mass, **more}


def listed():
    cases = [
        # the operator on the small lattice of the plain configuration: latency and launches
        ("operator_8", _case("operator", (8, 8, 8, 8), mass=-0.75)),
        # and on a production lattice
        ("operator_32", _case("operator", (32, 32, 32, 32), mass=-0.75)),
        # a two-index theory (d = 6) on an uneven lattice
        ("operator_sextet", _case("operator", (20, 10, 14, 12), repr="symmetric", mass=-0.3)),
        # the reference's solver on the small lattice
        ("cg_8", _case("cg", (8, 8, 8, 8), mass=-0.75, prec=1e-24)),
        # the pseudo-fermion solve of an HMC step, 16^3 x 32
        ("mixed_hmc", _case("mixed", (32, 16, 16, 16), mass=-0.75, prec=1e-24)),
        # the headline solve
        ("mixed_32", _case("mixed", (32, 32, 32, 32), mass=-0.75, prec=1e-24)),
        # twelve point-source propagators of a spectrum measurement
        ("multi_12", _case("multi", (32, 16, 16, 16), mass=-0.75, prec=1e-20, systems=12)),
        # RHMC in the SU(2) adjoint theory
        ("rational_adjoint", _case("rational", (48, 24, 24, 24), nc=2, repr="adjoint", mass=-0.3, prec=1e-20)),
        # one step of the Nf = 2 trajectory
        ("md_step", _case("md_step", (32, 16, 16, 16), mass=-0.55)),
        # an uneven batch of small lattices: this one, and two smaller ones
        ("lattices", _case("lattices", (16, 16, 16, 16), mass=-0.65, prec=1e-24, systems=3)),
        # the learned preconditioner and a step of its training
        ("network", _case("network", (32, 16, 16, 16), channels=8)),
        ("training", _case("training", (32, 16, 16, 16), channels=8)),
    ]
    return [{"name": n, **c} for n, c in cases]


def draw(rng):
    even = [4, 6, 8, 10, 12, 14, 16]

    def dims(most):
        """Even extents, at most `most` sites, the volume spread over its logarithm."""
        goal = math.exp(rng.uniform(math.log(8 ** 4 / 4), math.log(most)))
        d = sorted((rng.choice(even + [20, 24, 32]) for _ in range(4)), reverse=True)
        for _ in range(200):
            v = math.prod(d)
            i = rng.randrange(4)
            if v > min(most, 1.5 * goal):
                d[i] = max(4, d[i] - 2 if d[i] <= 16 else 16)
            elif v < goal / 1.5 and d[i] < 16:
                d[i] += 2
        return tuple(sorted(d, reverse=True))

    kind = rng.choice(["operator", "operator", "cg", "mixed", "multi", "rational", "md_step", "lattices", "network",
                       "training"])
    if kind == "operator":
        nc, rep, mass = rng.choice([(3, "fundamental", -0.7), (2, "adjoint", -0.3), (3, "symmetric", -0.3),
                                    (2, "fundamental", -0.6), (4, "antisymmetric", -0.3), (3, "adjoint", -0.2)])
        return _case("operator", dims(32 * 16 ** 3), nc=nc, repr=rep, mass=mass)
    if kind == "cg":
        return _case("cg", dims(12 ** 4), mass=rng.choice([-0.75, -0.5]), prec=rng.choice([1e-24, 1e-16]))
    if kind == "mixed":
        return _case("mixed", dims(32 * 16 ** 3), mass=rng.choice([-0.75, -0.6]), prec=rng.choice([1e-24, 1e-18]))
    if kind == "multi":
        return _case("multi", dims(16 ** 4), mass=rng.choice([-0.75, -0.6]), prec=1e-20,
                     systems=rng.choice([2, 3, 4, 6, 8, 12, 16]))
    if kind == "rational":
        return _case("rational", dims(32 * 16 ** 3), nc=2, repr="adjoint", mass=-0.3, prec=rng.choice([1e-20, 1e-14]))
    if kind == "md_step":
        return _case("md_step", dims(32 * 16 ** 3), mass=rng.choice([-0.55, -0.3]))
    if kind == "lattices":
        return _case("lattices", dims(12 ** 4), mass=-0.5, prec=1e-24, systems=rng.choice([2, 3, 4]))
    return _case(kind, dims(32 * 16 ** 3), channels=rng.choice([8, 16]))


# ------------------------------------------------------------------ gauge fields and sources
def _dims(case):
    return (case["t"], case["x"], case["y"], case["z"])


def _mul(a, b):
    """a @ b for many small matrices, as elementwise passes (quicker than a batched product)."""
    out = a[..., :, :1] * b[..., :1, :]
    for k in range(1, a.shape[-1]):
        out = torch.addcmul(out, a[..., :, k:k + 1], b[..., k:k + 1, :])
    return out


def _taylor_exp(a):
    e = torch.eye(a.shape[-1], dtype=a.dtype, device=a.device) + a
    t = a
    for k in range(2, 7):
        t = _mul(t, a) / k
        e = e + t
    return e


def _traceless_antihermitian(m):
    n = m.shape[-1]
    m = (m - m.mH) / 2
    return m - torch.diag_embed((m.diagonal(dim1=-2, dim2=-1).sum(-1) / n)[..., None].expand(*m.shape[:-2], n))


def _orthonormal(u):
    """Rows orthonormalised in order, the determinant's phase taken out of the last one."""
    rows = []
    for i in range(u.shape[-1]):
        r = u[..., i, :]
        for q in rows:
            r = r - (q.conj() * r).sum(-1, keepdim=True) * q
        rows.append(r / torch.linalg.vector_norm(r, dim=-1, keepdim=True))
    u = torch.stack(rows, -2)
    det = torch.linalg.det(u)
    last = u[..., -1:, :] * (det.conj() / det.abs())[..., None, None]
    return torch.cat([u[..., :-1, :], last], -2)


def _staples(u):
    """For every mu the sum V over nu of the two staples, U_mu(x) V_mu(x) being plaquettes."""
    out = []
    for mu in range(4):
        v = 0
        for nu in range(4):
            if nu == mu:
                continue
            n_mu = torch.roll(u[nu], -1, mu)
            v = v + _mul(n_mu, _mul(u[nu], torch.roll(u[mu], -1, nu)).mH)
            v = v + torch.roll(_mul(_mul(u[mu], n_mu).mH, u[nu]), 1, nu)
        out.append(v)
    return torch.stack(out)


@functools.lru_cache(maxsize=2)
def _links(dims, nc, seed):
    """(4, T, X, Y, Z, N, N) SU(N) links: a short Langevin run at the usual coupling."""
    beta = {2: 2.2, 3: 5.6, 4: 10.6}[nc]
    block = [min([k for k in range(8, n, 2) if n % k == 0], default=n) for n in dims]
    g = torch.Generator(DEVICE).manual_seed(1000 + seed)
    u = torch.eye(nc, dtype=torch.complex64, device=DEVICE).expand(4, *block, nc, nc).clone()
    for k in range(50):
        dt = 0.1 if k < 25 else 0.03 if k < 40 else 0.01
        drift = beta / (2 * nc) * _traceless_antihermitian(_mul(u, _staples(u)))
        # traceless anti-Hermitian noise, variance 1/2 per generator pair: sum_a i T_a xi_a
        xi = torch.randn(4, *block, nc, nc, dtype=torch.complex64, device=DEVICE, generator=g)
        noise = _traceless_antihermitian(xi)
        u = _mul(_taylor_exp(-dt * drift + math.sqrt(2 * dt) * noise), u)
        if k % 10 == 9:
            u = _orthonormal(u)
    u = _orthonormal(u.to(C128))
    return u.repeat(1, *(n // b for n, b in zip(dims, block)), 1, 1)


def _site_order(dims):
    """Lexicographic index of each site in the engine's order (even sites first)."""
    c = torch.meshgrid(*(torch.arange(n) for n in dims), indexing="ij")
    parity = (sum(c) % 2).reshape(-1)
    return torch.cat([torch.nonzero(parity == p).reshape(-1) for p in (0, 1)]).to(DEVICE)


def _host_links(u, dims):
    m = u.permute(1, 2, 3, 4, 0, 5, 6).reshape(-1, *u.shape[:1], *u.shape[-2:])[_site_order(dims)]
    return torch.stack([m.real, m.imag], 2).reshape(-1).cpu().numpy()


def _spinor(dims, d, seed, which=0):
    """Complex Gaussian field (T, X, Y, Z, 4, d) of unit variance."""
    g = torch.Generator(DEVICE).manual_seed(77 + 13 * seed + 1000003 * which)
    return torch.randn(*dims, 4, d, dtype=C128, device=DEVICE, generator=g)


def _host_spinor(psi, dims):
    """Spinor records re[d][4], im[d][4] in the engine's site order."""
    s = psi.reshape(-1, *psi.shape[-2:])[_site_order(dims)].transpose(1, 2)
    return torch.stack([s.real, s.imag], 1).reshape(-1).cpu().numpy()


class _Memory:
    """Device memory of a field for torch, which keeps this object, and with it the field and its lattice."""

    def __init__(self, field, shape):
        self.field = field
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (field.ptr, False), "version": 3}


def _even(lat, f):
    """The even sites of a device field, (spin * d + colour, site): a view, no copy."""
    v = torch.as_tensor(_Memory(f, (4 * lat.d, lat.Vh, 2)), device=DEVICE)
    return torch.view_as_complex(v)


def _lattice(case, seed, dims=None):
    dims = dims or _dims(case)
    lat = Lattice(dims, nc=case["nc"], repr=case["repr"], bc="antiperiodic", clover=True, csw=1.0)
    u = _links(tuple(dims), case["nc"], seed)
    lat.set_links(_host_links(u, dims))
    return lat


def _batch_dims(case):
    """The lattice of the case and smaller ones, every extent shrunk but even and at least 4."""
    out = []
    for k in range(case["systems"]):
        out.append(tuple(max(4, n * (case["systems"] - k) // case["systems"] // 2 * 2) for n in _dims(case)))
    return out


def _shapes(case):
    c = case["channels"]
    return [(9, c, 1, 4, 4), (9, c, c, 4, 4), (9, 1, c, 4, 4)]


def _weights(case, seed):
    """A network like a trained one: the identity on channel 0 plus mixing of every channel."""
    g = np.random.default_rng(seed)
    ws = []
    for shp in _shapes(case):
        w = 0.3 * (g.standard_normal(shp) + 1j * g.standard_normal(shp)) / math.sqrt(2 * 9 * 4 * shp[2])
        w[0, 0, 0] += np.eye(4)
        ws.append(w)
    return ws


def _training_pairs(case, seed):
    """(D e, e) on the even sites for errors e."""
    dims = _dims(case)
    ref = _Reference(_links(dims, case["nc"], seed), case["repr"])
    pairs = []
    for k in range(TRAINING_PAIRS):
        e = ref.even(_spinor(dims, 3, seed, 1 + k))
        pairs.append((ref.schur(case["mass"], e), e))
    return pairs


def prepare(case, seed):
    kind, dims = case["kind"], _dims(case)
    if kind == "lattices":
        solves = []
        for k, dk in enumerate(_batch_dims(case)):
            lat = _lattice(case, seed + k, dk)
            b = lat.field(_host_spinor(_spinor(dk, lat.d, seed, k), dk))
            solves.append((lat, case["mass"], case["prec"], lat.field(), b))
        return {"case": case, "solves": solves, "out": [_even(s[0], s[3]) for s in solves]}
    lat = _lattice(case, seed)
    s = {"case": case, "lat": lat}
    if kind in ("network", "training"):
        s["net"] = Ptc(lat, (1, case["channels"], case["channels"], 1))
        s["net"].set_weights(_weights(case, seed))
    if kind == "training":
        s["pairs"] = [tuple(lat.field(_host_spinor(f, dims)) for f in p) for p in _training_pairs(case, seed)]
        return s
    n = case.get("systems", 1)
    s["b"] = [lat.field(_host_spinor(_spinor(dims, lat.d, seed, k), dims)) for k in range(n)]
    s["x"] = [lat.field() for _ in range(n)]
    s["out"] = [_even(lat, x) for x in s["x"]]
    if kind == "md_step":
        lat.gauge_backup()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lattices":
        for lat, _, _, x, _ in state["solves"]:
            lat.spinor_zero(x)
        cg_inverter_lattices(state["solves"])
        return state["out"]
    lat, m = state["lat"], case["mass"]
    if kind == "training":
        return state["net"].gradient(state["pairs"])
    x, b = state["x"], state["b"]
    if kind == "operator":
        lat.Hphi_sq(m, x[0], b[0])
    elif kind == "cg":
        lat.spinor_zero(x[0])
        lat.cg_inverter("Hphi_sq", m, case["prec"], x[0], b[0])
    elif kind == "mixed":
        lat.spinor_zero(x[0])
        lat.cg_mixed("Hphi_sq", m, case["prec"], x[0], b[0])
    elif kind == "multi":
        for f in x:
            lat.spinor_zero(f)
        lat.cg_mixed_multi("Hphi_sq", m, case["prec"], x, b)
    elif kind == "rational":
        lat.rational_calc("Hphi_sq", m, case["prec"], A0, POLES, RESIDUES, x[0], b[0])
    elif kind == "network":
        state["net"].apply(x[0], b[0])
    elif kind == "md_step":
        # momenta from rest under every force, the links moved along them, and the operator
        # of the new field on the pseudo-fermion: what the next force evaluation starts with
        lat.gauge_restore()
        lat.represent_gauge_field()
        lat.zero_momenta()
        lat.improved_gauge_force(DT, 5.6, C0, (1 - C0) / 8)
        lat.begin_fermion_force()
        lat.wilson_fermion_force_q(DT, m, 1.0, b[0])
        lat.clover_logdet_force(m, 2.0)
        lat.end_fermion_force(DT)
        lat.update_links(DT)
        lat.represent_gauge_field()
        lat.Hphi(m, x[0], b[0])
        return {"kinetic": lat.momenta_action(), "field": state["out"][0]}
    return state["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def _site_counts(case, dims=None):
    d = {"fundamental": case["nc"], "adjoint": case["nc"] ** 2 - 1, "symmetric": case["nc"] * (case["nc"] + 1) // 2,
         "antisymmetric": case["nc"] * (case["nc"] - 1) // 2}[case["repr"]]
    return d, math.prod(dims or _dims(case)) // 2


def _operator_work(d, vh, real_bytes=8):
    """Bytes and operations of one Hphi: two hops over the half volume, both clover blocks."""
    matrices = (2 * 4 * 2 * d * d + 2 * 2 * (2 * d) ** 2) * real_bytes
    vectors = 2 * 8 * d * real_bytes
    hop = 8 * (8 * d * d * 2 + 4 * 2 * d) + 8 * d
    clover = 2 * 8 * (2 * d) ** 2
    return vh * (matrices + vectors), vh * 2 * (hop + clover)


#: CG iterations a solve takes on fields like these (they grow towards light quarks)
_ITERATIONS = {"cg": 200, "mixed": 250, "multi": 200, "rational": 42, "lattices": 120}


def work(case):
    kind = case["kind"]
    if kind == "lattices":
        flops = byts = 0
        for dk in _batch_dims(case):
            d, vh = _site_counts(case, dk)
            b, f = _operator_work(d, vh)
            flops += _ITERATIONS[kind] * (2 * f + vh * 8 * d * 10)
            byts += b
        return {"bytes": byts, "flops": flops}
    d, vh = _site_counts(case)
    b, f = _operator_work(d, vh)
    field = vh * 8 * d * 8
    if kind == "operator":
        return {"bytes": b, "flops": 2 * f}
    if kind == "cg":
        return {"bytes": b, "flops": _ITERATIONS[kind] * (2 * f + vh * 8 * d * 10)}
    if kind == "mixed":
        # per iteration: both matrices of the FP32 inner operator once per Hphi, the vectors once
        fb, _ = _operator_work(d, vh, 4)
        return {"bytes": _ITERATIONS[kind] * 2 * fb, "flops": _ITERATIONS[kind] * (2 * f + vh * 8 * d * 10)}
    if kind == "multi":
        fb, _ = _operator_work(d, vh, 4)
        return {"bytes": _ITERATIONS[kind] * 2 * fb,
                "flops": case["systems"] * _ITERATIONS[kind] * (2 * f + vh * 8 * d * 10)}
    if kind == "rational":
        n = len(POLES)
        return {"bytes": _ITERATIONS[kind] * (2 * b + 2 * n * field), "flops": _ITERATIONS[kind] * (2 * f + n * vh * 8 * d * 8)}
    if kind == "md_step":
        link = 2 * vh * 4 * 2 * 9 * 8
        mom = 2 * vh * 4 * 8 * 8
        # links read and written, momenta, clover term and inverse written, forces of 6 planes
        mm = 8 * 27
        flops = 2 * vh * 4 * (3 * (4 + 6 * 5 + 14) + 10) * mm + 2 * vh * 6 * 4 * 3 * mm
        return {"bytes": 4 * link + 4 * mom + 2 * 2 * vh * 2 * 36 * 8, "flops": flops}
    c = case["channels"]
    layers = 2 * vh * 9 * 3 * 8 * 16 * (c + c * c + c)
    act = 2 * vh * 96
    net = {"bytes": act * (1 + 4 * c + 1) + 3 * 2 * vh * 4 * 144, "flops": layers}
    if kind == "network":
        return net
    return {"bytes": TRAINING_PAIRS * 3 * net["bytes"], "flops": TRAINING_PAIRS * 3 * net["flops"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "operator":
        return {"rel": 1e-14, "max": 1e-12}
    if kind == "md_step":
        return {"rel": 1e-13, "max": 1e-11}
    if kind in ("network", "training"):
        return {"rel": 1e-2, "max": 0.2}
    # a solution is known to its residual times the square root of the condition number
    return {"rel": 100 * max(math.sqrt(case["prec"]), 1e-12)}


# ------------------------------------------------------------------ the definitions in plain torch
def _gammas(device):
    i = 1j
    g = torch.tensor([
        [[0, 0, -1, 0], [0, 0, 0, -1], [-1, 0, 0, 0], [0, -1, 0, 0]],
        [[0, 0, 0, -i], [0, 0, -i, 0], [0, i, 0, 0], [i, 0, 0, 0]],
        [[0, 0, 0, -1], [0, 0, 1, 0], [0, 1, 0, 0], [-1, 0, 0, 0]],
        [[0, 0, -i, 0], [0, 0, 0, i], [i, 0, 0, 0], [0, -i, 0, 0]]], dtype=C128, device=device)
    return g


def _su_generators(nc):
    """Anti-Hermitian generators with tr(t_a t_b) = -2 delta_ab, row by row."""
    out = []
    for r in range(nc):
        for c in range(nc):
            t = torch.zeros(nc, nc, dtype=C128)
            if r > c:
                t[r, c] = t[c, r] = 1j
            elif r < c:
                t[r, c], t[c, r] = 1, -1
            elif r > 0:
                v = math.sqrt(2 / (r * (r + 1)))
                for k in range(r):
                    t[k, k] = 1j * v
                t[r, r] = -1j * r * v
            else:
                continue
            out.append(t)
    return torch.stack(out)


def _basis(nc, rep):
    """Orthonormal basis of the representation space: N x N matrices."""
    if rep == "adjoint":
        return _su_generators(nc) * (-1j / math.sqrt(2))
    out = []
    for r in range(nc):
        for c in range(r + 1):
            b = torch.zeros(nc, nc, dtype=C128)
            if rep == "symmetric" and r == c:
                b[r, r] = 1
            elif r != c:
                b[r, c] = b[c, r] = 1 / math.sqrt(2)
                if rep == "antisymmetric":
                    b[r, c] *= -1
            else:
                continue
            out.append(b)
    return torch.stack(out)


class _Reference:
    """The even-odd Wilson-clover operator of a gauge field (4, T, X, Y, Z, N, N)."""

    def __init__(self, u, rep, csw=1.0):
        self.device = u.device
        self.dims = tuple(u.shape[1:5])
        self.rep, self.nc = rep, u.shape[-1]
        self.gamma = _gammas(u.device)
        self.g5 = torch.diag(torch.tensor([1, 1, -1, -1], dtype=C128, device=u.device))
        t = torch.arange(self.dims[0], device=u.device).view(-1, 1, 1, 1, 1, 1)
        links = [self._map(u[mu]) for mu in range(4)]
        self.u = [torch.where(t == 0, -links[0], links[0])] + links[1:]
        self.d = links[0].shape[-1]
        self.clover = self._clover(u, csw)
        self._inverse = {}
        c = torch.meshgrid(*(torch.arange(n, device=u.device) for n in self.dims), indexing="ij")
        self.parity = (sum(c) % 2)[..., None, None]

    def _map(self, u):
        if self.rep == "fundamental":
            return u
        b = _basis(self.nc, self.rep).to(u.device)
        w = u.mH if self.rep == "adjoint" else u.transpose(-1, -2)
        ub = torch.einsum("...ij,mjk,...kl->...mil", u, b, w)
        r = torch.einsum("nil,...mil->...nm", b.conj(), ub)
        return r.real.to(C128) if self.rep == "adjoint" else r

    def _clover(self, u, csw):
        """-csw/16 sum_{mu<nu} sigma_mu_nu F_mu_nu, (T, X, Y, Z, 4, d, 4, d)."""
        out = 0
        for mu in range(4):
            for nu in range(mu + 1, 4):
                a, b = u[mu], u[nu]
                fm, fn = torch.roll(b, -1, mu), torch.roll(a, -1, nu)       # U_nu(x+mu), U_mu(x+nu)
                p1 = a @ fm @ (b @ fn).mH                                     # at x
                bm, am = torch.roll(b, 1, mu), torch.roll(a, 1, mu)         # U_nu(x-mu), U_mu(x-mu)
                amn = torch.roll(fn, 1, mu)                                   # U_mu(x-mu+nu)
                p2 = b @ (bm @ amn).mH @ am
                bn, an = torch.roll(b, 1, nu), torch.roll(a, 1, nu)         # U_nu(x-nu), U_mu(x-nu)
                bmn, amnn = torch.roll(bm, 1, nu), torch.roll(am, 1, nu)    # at x-mu-nu
                p3 = (bmn @ am).mH @ amnn @ bn
                bpm = torch.roll(fm, 1, nu)                                   # U_nu(x+mu-nu)
                p4 = bn.mH @ an @ bpm @ a.mH
                q = sum(self._map(p) for p in (p1, p2, p3, p4))
                f = -1j * (q - q.mH)
                sigma = 0.5j * (self.gamma[mu] @ self.gamma[nu] - self.gamma[nu] @ self.gamma[mu])
                out = out + torch.einsum("st,...ab->...satb", -csw / 16 * sigma, f)
        return out

    def even(self, psi):
        return torch.where(self.parity == 0, psi, 0)

    def odd(self, psi):
        return torch.where(self.parity == 1, psi, 0)

    def hop(self, psi):
        """-1/2 sum_mu [(1 - g_mu) U psi(x+mu) + (1 + g_mu) U^dag psi(x-mu)]"""
        out = 0
        one = torch.eye(4, dtype=C128, device=self.device)
        for mu in range(4):
            f = torch.roll(psi, -1, mu) @ self.u[mu].transpose(-1, -2)
            b = torch.roll(psi @ self.u[mu].conj(), 1, mu)
            out = out - 0.5 * ((one - self.gamma[mu]) @ f + (one + self.gamma[mu]) @ b)
        return out

    def site(self, m, psi):
        n = 4 * self.d
        a = self.clover.reshape(*self.dims, n, n) @ psi.reshape(*self.dims, n, 1)
        return (4 + m) * psi + a.reshape(psi.shape)

    def site_inverse(self, m, psi):
        """Chirality by chirality: sigma F does not mix the upper and lower spins."""
        n = 2 * self.d
        out = []
        for k, s in enumerate((slice(0, 2), slice(2, 4))):
            if (m, k) not in self._inverse:
                a = self.clover[..., s, :, s, :].reshape(*self.dims, n, n)
                eye = torch.eye(n, dtype=C128, device=self.device)
                self._inverse[m, k] = torch.linalg.inv(a + (4 + m) * eye)
            out.append((self._inverse[m, k] @ psi[..., s, :].reshape(*self.dims, n, 1)).reshape(psi[..., s, :].shape))
        return torch.cat(out, -2)

    def schur(self, m, psi):
        psi = self.even(psi)
        return self.even(self.site(m, psi) - self.hop(self.site_inverse(m, self.odd(self.hop(psi)))))

    def h(self, m, psi):
        return self.g5 @ self.schur(m, psi)

    def h_sq(self, m, psi):
        return self.h(m, self.h(m, psi))

    def device_even(self, psi):
        """Even sites as the engine's fields hold them."""
        order = _site_order(self.dims)
        half = order[:order.numel() // 2]
        return psi.reshape(-1, 4 * self.d)[half].T.contiguous()

    def transport(self, f, p):
        """f (T, X, Y, Z, C, 4, 3) carried to every site along one of the nine paths."""
        if p == 0:
            return f
        mu = (p - 1) % 4
        u = self.u[mu].unsqueeze(4)
        if p <= 4:
            return torch.roll(f, -1, mu) @ u.transpose(-1, -2)
        return torch.roll(f @ u.conj(), 1, mu)


def _solve(ref, m, b, shift=0.0, most=4000):
    """Conjugate gradient to the floor of double precision, restarted once."""
    x = torch.zeros_like(b)
    bb = b.norm().item()
    for _ in range(2):
        r = b - (ref.h_sq(m, x) + shift * x)
        p, rr = r.clone(), r.norm().item() ** 2
        for _ in range(most):
            if math.sqrt(rr) < 1e-15 * bb:
                break
            q = ref.h_sq(m, p) + shift * p
            a = rr / torch.sum(p.conj() * q).real.item()
            x = x + a * p
            r = r - a * q
            new = r.norm().item() ** 2
            p, rr = r + (new / rr) * p, new
    return x


def _gauge_action(u, beta, c0):
    c1 = (1 - c0) / 8
    total = 0
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            a, b = u[mu], u[nu]
            b1, a1 = torch.roll(b, -1, mu), torch.roll(a, -1, nu)
            if mu < nu:
                total = total + c0 * torch.sum((a @ b1) * (b @ a1).conj()).real
            # two steps along mu, one along nu
            aa = a @ torch.roll(a, -1, mu)
            total = total + c1 * torch.sum((aa @ torch.roll(b, -2, mu)) * (b @ torch.roll(aa, -1, nu)).conj()).real
    return -beta / u.shape[-1] * total


def _md_step(case, seed):
    dims, m = _dims(case), case["mass"]
    u0 = _links(dims, 3, seed)
    gens = _su_generators(3).to(u0.device)
    phi = _spinor(dims, 3, seed, 0)
    w = torch.zeros(4, *dims, 8, dtype=torch.float64, device=u0.device, requires_grad=True)
    a = torch.einsum("...a,aij->...ij", w.to(C128), gens)
    u = u0 + a @ u0                                    # exp(a) u0 to first order: the derivative at 0
    ref = _Reference(u, "fundamental")
    x = ref.even(phi)
    hx = ref.h(m, x).detach()
    pseudo = torch.sum(hx.conj() * ref.h(m, x)).real
    n = 6
    det = 0
    for s in (slice(0, 2), slice(2, 4)):
        c = ref.clover[..., s, :, s, :].reshape(*dims, n, n) + (4 + m) * torch.eye(n, dtype=C128, device=u0.device)
        det = det + torch.where(ref.parity[..., 0, 0] == 1, torch.linalg.slogdet(c)[1], 0).sum()
    total = -0.5 * _gauge_action(u, 5.6, C0) + pseudo + det
    force, = torch.autograd.grad(total, w)
    mom = DT * force
    u1 = torch.linalg.matrix_exp(DT * torch.einsum("...a,aij->...ij", mom.to(C128), gens)) @ u0
    new = _Reference(u1, "fundamental")
    return {"kinetic": float((mom ** 2).sum()), "field": new.device_even(new.h(m, x))}


def _network(ref, ws, f, keep=False):
    acts = [f[..., None, :, :]]
    for w in ws:
        out = 0
        for p in range(9):
            out = out + torch.einsum("oist,...ita->...osa", w[p], ref.transport(acts[-1], p))
        acts.append(out)
    return acts[-1][..., 0, :, :]


def exact(case, seed):
    kind, dims = case["kind"], _dims(case)
    if kind == "lattices":
        out = []
        for k, dk in enumerate(_batch_dims(case)):
            ref = _Reference(_links(dk, case["nc"], seed + k), case["repr"])
            out.append(ref.device_even(_solve(ref, case["mass"], ref.even(_spinor(dk, ref.d, seed, k)))))
        return out
    if kind == "md_step":
        return _md_step(case, seed)
    sites = math.prod(dims)
    if (kind in ("mixed", "rational") and sites > 40000) or (kind == "multi" and sites * case["systems"] > 40000):
        return None
    ref = _Reference(_links(dims, case["nc"], seed), case["repr"])
    m = case["mass"]
    if kind in ("network", "training"):
        ws = [torch.from_numpy(w).to(ref.device) for w in _weights(case, seed)]
        if kind == "network":
            return [ref.device_even(ref.even(_network(ref, ws, ref.even(_spinor(dims, 3, seed, 0)))))]
        for w in ws:
            w.requires_grad_(True)
        grads, loss = [np.zeros(s, dtype=complex) for s in _shapes(case)], 0.0
        for r, e in _training_pairs(case, seed):
            part = torch.sum((ref.even(_network(ref, ws, r)) - e).abs() ** 2) / torch.sum(e.abs() ** 2)
            for g, t in zip(grads, torch.autograd.grad(part, ws)):
                g += 0.5 * t.resolve_conj().cpu().numpy()          # d / d conj(W)
            loss += part.item()
        return loss, grads
    b = [ref.even(_spinor(dims, ref.d, seed, k)) for k in range(case.get("systems", 1))]
    if kind == "operator":
        return [ref.device_even(ref.h_sq(m, b[0]))]
    if kind == "rational":
        x = A0 * b[0]
        for p, r in zip(POLES, RESIDUES):
            x = x + r * _solve(ref, m, b[0], shift=p)
        return [ref.device_even(x)]
    return [ref.device_even(_solve(ref, m, f)) for f in b]
