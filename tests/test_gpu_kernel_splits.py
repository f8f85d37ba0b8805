"""The work splits of the FP64 kernels where they change over or leave remainders: four lanes a site up
to kQuadSites = 4736 output sites and one thread a site above (d <= 6), blocks of 32 sites of the force
and clover kernels with a ragged last block, and both splits of the persistent CG.  Against the FP64
oracle; 1e-13 relative as in the parity tests of these functions (sums of a few hundred terms of
relative rounding 1.1e-16)."""
import numpy as np
import pytest

from tests.helpers import make_pair, rel, source

pytestmark = pytest.mark.gpu
TOL = 1e-13
ABOVE = (8, 10, 10, 12)          # 4800 even sites: one thread a site, a ragged last block of 128
BELOW = (2, 6, 6, 6)             # 216 even sites: four lanes a site, 13.5 blocks of 32 sites


@pytest.mark.parametrize("dims", [ABOVE, BELOW])
@pytest.mark.parametrize("name", ["su3_fund_ap", "su2_adj_ap", "su4_fund_ap", "su3_sym_ap", "su3_fund_open",
                                  "su3_fund_ap_nocl", "su3_fund_ap_full"])
def test_operator(name, dims):
    if name == "su3_fund_open" and dims[0] < 4:
        dims = (4, 6, 6, 6)
    lat, O, rng = make_pair(name, dims, seed=21)
    src = source(O, rng)
    for fn, args in (("Dphi", [-0.6]), ("Hphi_sq", [-0.4])):
        s, d = lat.field(src), lat.field()
        s2, d2 = src.copy(), O.new_field()
        getattr(lat, fn)(*args, d, s)
        getattr(O, fn)(*args, d2, s2)
        assert rel(lat.download(d), d2) < TOL
        assert rel(lat.download(s), s2) < TOL
    if O.p.clover and O.p.eo:
        lo = O.compute_ldl(4 - 0.4)
        assert rel(lat.ldl(-0.4)[O.Vh:], lo[O.Vh:]) < TOL


@pytest.mark.parametrize("name", ["su3_fund_ap", "su2_adj_ap", "su4_fund_ap", "su3_sym_ap", "su3_adj_ap", "su3_fund_sf"])
def test_forces_ragged(name):
    dims = (6, 2, 6, 6) if name.endswith("sf") else BELOW
    lat, O, rng = make_pair(name, dims, seed=22)
    a0, b0 = source(O, rng), source(O, rng)
    a, b = lat.field(a0), lat.field(b0)
    lat.zero_momenta()
    O.mom[:] = 0
    lat.begin_fermion_force()
    O.begin_fermion_force()
    lat.wilson_fermion_force_q_multi(0.1, -0.5, [0.7, -0.2], [a, b])
    for f, w in ((a0, 0.7), (b0, -0.2)):
        O.wilson_fermion_force_q(0.1, -0.5, w, f.copy())
    lat.clover_logdet_force(-0.5, 2.0)
    O.clover_logdet_force(-0.5, 2.0)
    assert rel(lat.clover_force(), O.cl_force, floor=1.0) < TOL
    lat.end_fermion_force(0.1)
    O.end_fermion_force(0.1)
    lat.improved_gauge_force(0.1, 5.6, 5.0 / 3.0, -1.0 / 12.0)
    O.improved_gauge_force(0.1, 5.6, 5.0 / 3.0, -1.0 / 12.0)
    lat.wilson_gauge_force(0.05, 5.6)
    O.wilson_gauge_force(0.05, 5.6)
    assert rel(lat.momenta(), O.mom, floor=1.0) < TOL
    assert rel(lat.clover_term(), O.cl_term, floor=1.0) < TOL


@pytest.mark.parametrize("name,dims", [("su3_fund_ap", ABOVE), ("su3_fund_ap", BELOW), ("su3_fund_ap_nocl", BELOW),
                                       ("su3_sym_ap", BELOW), ("su2_fund_ap", (4, 4, 4, 6)), ("su2_fund_ap", ABOVE),
                                       ("su4_fund_ap", BELOW), ("su4_fund_ap", ABOVE)])
def test_persistent_cg(name, dims):
    """One lattice per call of cg_inverter: the true residual meets prec and the solution is the
    oracle's CG's (both solve to 1e-11 of |b|; the operator's condition number here is below 1e4)."""
    lat, O, rng = make_pair(name, dims, seed=23)
    b0 = source(O, rng)
    b, x = lat.field(b0), lat.field()
    it = lat.cg_inverter("Hphi_sq", 0.2, 1e-22, x, b)
    xo = O.new_field()
    ito = O.cg("Hphi_sq", 0.2, 1e-22, xo, b0.copy())
    ito = ito[0] if isinstance(ito, tuple) else ito
    assert abs(it - ito) <= 1
    assert rel(lat.download(x)[:O.Vh], xo[:O.Vh]) < 1e-7
    q = O.new_field()
    xs = lat.download(x)
    O.Hphi_sq(0.2, q, xs)
    r = (q - b0)[:O.Vh]
    assert np.vdot(r, r).real < 4e-22 * np.vdot(b0[:O.Vh], b0[:O.Vh]).real
    # a call that starts from the solution makes no iteration, and maxiter ends a solve early
    assert lat.cg_inverter("Hphi_sq", 0.2, 1e-20, x, b) == 0
    lat.spinor_zero(x)
    assert lat.cg_inverter("Hphi_sq", 0.2, 1e-22, x, b, maxiter=3) == 3 and lat.last_status == 4


@pytest.mark.parametrize("channels", [(1, 8, 8, 1), (1, 16, 16, 1)])
def test_network_on_ragged_tiles(channels):
    """432 even sites: 6.75 tiles of 64, so one tile straddles the parities and takes all nine paths,
    the others leave out the paths that carry nothing.  BF16 operands: 2e-2 as in the layer tests."""
    from oracle import ptc_oracle as po
    from yahmc_b200 import Ptc
    lat, O, rng = make_pair("su3_fund_ap", (4, 6, 6, 6), seed=24)
    net = Ptc(lat, channels)
    Ws = [(rng.standard_normal(s) + 1j * rng.standard_normal(s)) / np.sqrt(2 * 9 * 4 * s[2]) for s in net.shapes()]
    net.set_weights(Ws)
    pairs = []
    for _ in range(2):
        r, e = source(O, rng), source(O, rng)
        r[O.Vh:] = 0
        e[O.Vh:] = 0
        pairs.append((r, e))
    onet = po.Net(Ws)
    d, s = lat.field(), lat.field(pairs[0][0])
    net.apply(d, s)
    assert rel(lat.download(d)[:O.Vh], po.apply_even(O, onet, pairs[0][0][:O.Vh])) < 2e-2
    loss, grads = net.gradient([(lat.field(r), lat.field(e)) for r, e in pairs])
    lo, go = po.loss_and_grads(O, onet, [(r[:O.Vh], e[:O.Vh]) for r, e in pairs])
    assert abs(loss - lo) < 2e-2 * lo
    for g, h in zip(grads, go):
        assert rel(g, h) < 2e-2


@pytest.mark.parametrize("name,dims", [("su4_asym_ap", BELOW), ("su3_adj_ap", BELOW), ("su4_sym_ap", BELOW),
                                       ("su4_sym_ap", (10, 10, 10, 12)), ("su4_adj_ap", (2, 4, 4, 6))])
def test_clover_term(name, dims):
    """A warp per plane up to d = 8 (blocks of 32 sites, the last one ragged), a thread a site above, with
    leaves as chains (d = 10 below 10000 sites) or as pairs of products."""
    lat, O, rng = make_pair(name, dims, seed=25)
    assert rel(lat.clover_term(), O.cl_term, floor=1.0) < TOL
    assert rel(lat.repr_links(), O.links) < TOL


@pytest.mark.parametrize("name,dims", [
    ("su2_asym_ap", (24, 16, 16, 14)), ("su2_fund_ap", BELOW), ("su3_fund_ap", (4, 4, 4, 4)),
    ("su3_fund_ap", (14, 12, 12, 12)), ("su3_fund_ap", (16, 12, 12, 12)),
    ("su4_fund_ap", BELOW), ("su4_fund_ap", (16, 14, 12, 12)), ("su4_fund_ap", (24, 16, 16, 14)),
    ("su3_sym_ap", BELOW), ("su3_sym_ap", (16, 14, 12, 12)),
    ("su3_adj_ap", BELOW), ("su4_sym_ap", BELOW), ("su4_adj_ap", (2, 4, 4, 6))])
def test_fermion_forces_one_and_several_poles(name, dims):
    """The hopping force of one pole and of three (with and without the pole loop; the spinors of a pole
    at once or in pairs), and the clover force's three splits (warps on small lattices, a thread a site or
    per site and slot above), on both sides of the changes at 10000 to 80000 sites.  The large
    lattices compare a call of three poles with the oracle's sum on a third of the work: three calls of one
    pole must give the same, and one of them is the oracle's."""
    lat, O, rng = make_pair(name, dims, seed=26)
    fields_ = [source(O, rng) for _ in range(3)]
    dev = [lat.field(f) for f in fields_]
    w = (0.7, -0.2, 0.35)
    first = None
    lat.zero_momenta()
    lat.begin_fermion_force()
    for f, c in zip(dev, w):
        lat.wilson_fermion_force_q(0.1, -0.5, c, f)
        if first is None:
            first = lat.clover_force().copy(), lat.momenta().copy()
    O.mom[:] = 0
    O.begin_fermion_force()
    O.wilson_fermion_force_q(0.1, -0.5, w[0], fields_[0].copy())
    assert rel(first[0], O.cl_force, floor=1.0) < TOL
    assert rel(first[1], O.mom, floor=1.0) < TOL
    one = lat.clover_force().copy(), lat.momenta().copy()
    lat.zero_momenta()
    lat.begin_fermion_force()
    lat.wilson_fermion_force_q_multi(0.1, -0.5, list(w), dev)
    assert rel(lat.clover_force(), one[0], floor=1.0) < TOL
    assert rel(lat.momenta(), one[1], floor=1.0) < TOL
