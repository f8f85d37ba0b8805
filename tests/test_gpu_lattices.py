"""Independent CG solves on several lattices at once (yg_cg_inverter_lattices).

Hphi_sq solves on even-odd lattices of one representation dimension (2, 3, 4 or 6), all with
or all without a clover term and without open/SF boundaries, run as one persistent kernel:
each lattice's whole cg_inverter loop (cg.cpp:132-202) runs on a group of blocks with
bounded barriers.  Small systems of cg_inverter itself take the same kernel, so the persistent
solves are compared with the recurrence launch by launch (engine operator and BLAS), reached
through a batch too large for persistent solves: its reductions add the same terms in another
order, so solutions agree to rounding (relative 1e-10) and iteration counts within one.  Any other
mix runs each lattice's cg_inverter in its own host thread and must match one-at-a-time calls bit
for bit."""
import numpy as np
import pytest

from tests.helpers import make_pair, source

pytestmark = pytest.mark.gpu


_filler = []


def _launch_by_launch(lat, mass, prec, b, maxiter=0):
    """cg_inverter's recurrence with one launch per step: the lattice in a batch with one of 165888
    colours and open boundaries (one iteration), which runs on host threads without the persistent
    kernel.  Returns the solution on the host and the iteration count."""
    from yahmc_b200 import Lattice, cg_inverter_lattices
    if not _filler:
        big = Lattice((24, 16, 16, 18), bc="open", clover=False)
        _filler.extend([big, big.field(), big.field(np.ones((big.V, 4, big.d)) + 0j)])
    x = lat.field()
    its, rc, path = cg_inverter_lattices([(lat, mass, prec, x, b, maxiter), (_filler[0], 0.5, 1e-30, *_filler[1:], 1)],
                                         with_path=True)
    assert path == 0 and rc == 4 and its[1] == 1
    return lat.download(x), its[0]


def _one_call(lat, mass, prec, b):
    x = lat.field()
    it = lat.cg_inverter("Hphi_sq", mass, prec, x, b)
    return lat.download(x), it


def _setup(case, mass=-0.4, prec=1e-22, reference=_launch_by_launch):
    solves, refs = [], []
    for k, (name, dims) in enumerate(case):
        lat, O, rng = make_pair(name, dims, seed=90 + k)
        b = lat.field(source(O, rng))
        refs.append(reference(lat, mass, prec, b))
        solves.append((lat, mass, prec, lat.field(), b, 0))
    return solves, refs


def _even(lat, f):
    return lat.download(f)[:lat.V // 2]


PERSISTENT = [
    [("su3_fund_ap", (8, 8, 8, 8)), ("su3_fund_ap", (12, 12, 12, 12)), ("su3_fund_ap", (16, 16, 16, 16))],
    [("su2_adj_ap", (4, 6, 4, 8)), ("su3_fund_ap", (8, 8, 8, 8)), ("su3_fund_per", (6, 4, 4, 4))],
    [("su3_fund_ap_nocl", (12, 8, 8, 8)), ("su3_fund_ap_nocl", (4, 4, 4, 4))],
    [("su2_fund_ap", (8, 8, 8, 8)), ("su2_fund_ap", (4, 4, 4, 6))],
    [("su4_fund_ap", (8, 4, 4, 4)), ("su4_fund_ap", (4, 4, 4, 4))],
    [("su3_sym_ap", (4, 4, 4, 4)), ("su4_asym_ap", (6, 4, 4, 4))],
    [("su2_fund_ap", (10, 10, 10, 10)), ("su2_fund_ap", (4, 4, 4, 6))],          # a thread a site
    [("su4_fund_ap", (8, 10, 10, 12)), ("su4_fund_ap", (4, 4, 4, 4))],
    [("su3_fund_ap", (16, 16, 16, 14)), ("su3_fund_per", (16, 16, 16, 16))],       # two tiles a block
]


@pytest.mark.parametrize("case", PERSISTENT)
def test_persistent_batch_matches_one_at_a_time(case):
    from yahmc_b200 import cg_inverter_lattices
    solves, refs = _setup(case)
    for _ in range(2):                                   # twice: scratch fields and buffers reused
        for s in solves:
            s[0].spinor_zero(s[3])
        its, rc, path = cg_inverter_lattices(solves, with_path=True)
        assert rc == 0 and path == 1
        for (lat, _, _, x, _, _), (xr, itr), it in zip(solves, refs, its):
            assert abs(it - itr) <= 1, (it, itr)
            got, ref = _even(lat, x), xr[:lat.V // 2]
            assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


def test_persistent_batch_maxiter_and_converged_start():
    """A lattice that stops at maxiter reports YG_MAXITER and exactly maxiter iterations; a
    lattice whose initial guess already meets prec reports 0 iterations (cg.cpp:151-153), as
    cg_inverter does; the others are unaffected."""
    from yahmc_b200 import cg_inverter_lattices
    case = [("su3_fund_ap", (8, 8, 8, 8)), ("su3_fund_ap", (12, 8, 8, 8)), ("su3_fund_ap", (4, 4, 4, 4))]
    solves, refs = _setup(case)
    lat0, m, p, x0, b0, _ = solves[0]
    solves[0] = (lat0, m, p, x0, b0, 7)                  # stops after 7 iterations
    lat2, _, _, x2, b2, _ = solves[2]
    lat2.upload(x2, refs[2][0])                          # starts at a solution to 1e-22 ...
    solves[2] = (lat2, m, 1e-16, x2, b2, 0)              # ... of a system asked for 1e-16
    lat0.spinor_zero(x0)
    solves[1][0].spinor_zero(solves[1][3])
    its, rc, path = cg_inverter_lattices(solves, with_path=True)
    assert path == 1 and rc == 4
    assert its[0] == 7
    assert abs(its[1] - refs[1][1]) <= 1
    assert its[2] == lat2.cg_inverter("Hphi_sq", m, 1e-16, lat2.field(refs[2][0]), b2) == 0
    x7, it7 = _launch_by_launch(lat0, m, p, b0, maxiter=7)
    assert it7 == 7
    assert lat0.cg_inverter("Hphi_sq", m, p, lat0.field(), b0, maxiter=7) == 7
    a, c = _even(lat0, x0), x7[:lat0.V // 2]
    assert np.abs(a - c).max() <= 1e-10 * np.abs(c).max()


def test_persistent_batch_wait_limit_returns_timeout():
    """A barrier wait limit of a few cycles runs out at the first barrier: the kernel returns
    (no trap, no hang), the call reports YG_TIMEOUT, and the next call on the same lattices
    solves them normally."""
    from yahmc_b200 import cg_inverter_lattices
    case = [("su3_fund_ap", (8, 8, 8, 8)), ("su3_fund_ap", (16, 16, 16, 16))]
    solves, refs = _setup(case)
    its, rc, path = cg_inverter_lattices(solves, wait_cycles=8, with_path=True)
    assert path == 1 and rc == 7
    for s in solves:
        s[0].spinor_zero(s[3])
    its, rc = cg_inverter_lattices(solves)
    assert rc == 0
    for (lat, _, _, x, _, _), (xr, itr), it in zip(solves, refs, its):
        assert abs(it - itr) <= 1
        got, ref = _even(lat, x), xr[:lat.V // 2]
        assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("case", [
    [("su3_fund_open", (8, 8, 8, 8)), ("su2_adj_ap", (4, 6, 4, 8)), ("su3_fund_ap_full", (8, 8, 8, 8)),
     ("su3_fund_ap_nocl", (12, 8, 8, 8))],
    [("su3_adj_ap", (4, 4, 4, 4)), ("su3_adj_ap", (6, 4, 4, 4))],          # d = 8: host threads
])
def test_threads_equal_sequential(case):
    from yahmc_b200 import cg_inverter_lattices
    solves, refs = _setup(case, reference=_one_call)
    for _ in range(2):
        for s in solves:
            s[0].spinor_zero(s[3])
        its, rc, path = cg_inverter_lattices(solves, with_path=True)
        assert rc == 0 and path == 0
        for (lat, _, _, x, _, _), (xr, itr), it in zip(solves, refs, its):
            assert it == itr
            assert np.array_equal(lat.download(x), xr)


def test_errors():
    from yahmc_b200 import YGError, cg_inverter_lattices
    lat, O, rng = make_pair("su3_fund_ap", (8, 8, 8, 8), seed=99)
    b = lat.field(source(O, rng))
    with pytest.raises(YGError):
        cg_inverter_lattices([(lat, -0.4, 1e-20, lat.field(), b), (lat, -0.4, 1e-20, lat.field(), b)])


def test_persistent_solve_goes_on_over_several_launches():
    """One launch makes at most 1000 iterations: an ill-conditioned system (smallest eigenvalues of
    Hphi_sq near 1e-6 on random links) needs more, so the solve goes on in further launches, and ends where
    its true residual meets prec, or at exactly maxiter."""
    from yahmc_b200 import cg_inverter_lattices, launch_count
    lat, O, rng = make_pair("su3_fund_ap", (4, 4, 4, 4), seed=23)
    b0 = source(O, rng)
    b, x = lat.field(b0), lat.field()
    lat.cg_inverter("Hphi_sq", -2.3, 1e-14, x, b, maxiter=10)
    lat.spinor_zero(x)
    n0 = launch_count()
    assert lat.cg_inverter("Hphi_sq", -2.3, 1e-14, x, b, maxiter=10) == 10
    n10 = launch_count() - n0
    lat.spinor_zero(x)
    n0 = launch_count()
    it = lat.cg_inverter("Hphi_sq", -2.3, 1e-14, x, b)
    assert it > 2000
    assert launch_count() - n0 == n10 + (it - 1) // 1000
    q, xs = O.new_field(), lat.download(x)
    O.Hphi_sq(-2.3, q, xs)
    r = (q - b0)[:O.Vh]
    # the recursive residual meets prec; the true one differs by the rounding of A x: 1.1e-16 times the
    # largest eigenvalue (below 100) times |x| (2e5 |b| here), 2e-9 |b|, so by 2 * 1e-7 * 2e-9 |b|^2 at most
    assert np.vdot(r, r).real < 1.1e-14 * np.vdot(b0[:O.Vh], b0[:O.Vh]).real
    # a batch in which one lattice ends in the first launch and one stops at maxiter in the third
    lat2, O2, rng2 = make_pair("su3_fund_ap", (4, 4, 4, 6), seed=24)
    b2, x2 = lat2.field(source(O2, rng2)), lat2.field()
    x2s, it2 = _launch_by_launch(lat2, 0.2, 1e-22, b2)
    lat.spinor_zero(x)
    its, rc, path = cg_inverter_lattices([(lat, -2.3, 0.0, x, b, 2345), (lat2, 0.2, 1e-22, x2, b2)], with_path=True)
    assert path == 1 and rc == 4 and its[0] == 2345 and abs(its[1] - it2) <= 1
    got, ref = _even(lat2, x2), x2s[:lat2.V // 2]
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


def test_persistent_batch_of_one_large_and_many_tiny_lattices():
    """63 lattices of 8 even sites beside one of 384 tiles: a block for each tiny lattice and the
    large one's share stay within the resident grid."""
    from yahmc_b200 import Lattice, cg_inverter_lattices
    big = Lattice((24, 16, 16, 16))
    big.momenta_gaussian(5)
    big.update_links(0.3)
    big.represent_gauge_field()
    bb = big.field(np.random.default_rng(6).standard_normal((big.V, 4, big.d)) + 0j)
    tiny = [make_pair("su3_fund_ap", (2, 2, 2, 2), seed=200 + k) for k in range(63)]
    tb = [lat.field(source(O, rng)) for lat, O, rng in tiny]
    solves = [(big, 0.5, 1e-20, big.field(), bb)]
    solves += [(lat, 0.5, 1e-20, lat.field(), b) for (lat, _, _), b in zip(tiny, tb)]
    its, rc, path = cg_inverter_lattices(solves, with_path=True)
    assert rc == 0 and path == 1
    for k, (lat, m, prec, x, b) in enumerate(solves):
        ref = lat.field()
        itr = lat.cg_inverter_multi("Hphi_sq", m, prec, [ref], [b])[0]
        assert abs(its[k] - itr) <= 1
        got, want = _even(lat, x), _even(lat, ref)
        assert np.abs(got - want).max() <= 1e-9 * np.abs(want).max()


def test_host_threads_share_the_device():
    """Calls of cg_inverter from several host threads on lattices of their own run at once as far as
    their blocks fit, and give the bits of one call after the other.  8^4 takes 64 of 444 slots: six
    threads at once are quicker than six calls in a row (measured 2.3 against 8 ms)."""
    import threading
    import time
    case = [("su3_fund_ap", (8, 8, 8, 8))] * 6
    solves = []
    for k, (name, dims) in enumerate(case):
        lat, O, rng = make_pair(name, dims, seed=300 + k)
        solves.append((lat, lat.field(source(O, rng)), lat.field(), lat.field()))

    def one(s, x):
        lat, b, _, _ = s
        lat.cg_inverter("Hphi_sq", -0.4, 1e-22, x, b, maxiter=400)

    def all_at_once():
        th = [threading.Thread(target=one, args=(s, s[3])) for s in solves]
        for t in th:
            t.start()
        for t in th:
            t.join()

    def one_by_one():
        for s in solves:
            one(s, s[2])

    times = {}
    for name, run, slot in (("row", one_by_one, 2), ("threads", all_at_once, 3)):
        best = 1e9
        for _ in range(4):
            for s in solves:
                s[0].spinor_zero(s[slot])
                s[0].synchronize()
            t = time.perf_counter()
            run()
            best = min(best, time.perf_counter() - t)
        times[name] = best
    for s in solves:
        assert np.array_equal(_even(s[0], s[2]), _even(s[0], s[3]))
    assert times["threads"] < 0.8 * times["row"], times


@pytest.mark.parametrize("name", ["su3_fund_ap", "su4_fund_ap", "su3_sym_ap", "su2_fund_ap", "su3_fund_ap_nocl"])
def test_launch_by_launch_against_oracle(name):
    """The recurrence launch by launch, the reference of the tests above, is the oracle's (both solve to
    1e-11 of |b|; the condition number of the operator is below 1e4)."""
    lat, O, rng = make_pair(name, (4, 4, 4, 6), seed=77)
    b0 = source(O, rng)
    x, it = _launch_by_launch(lat, 0.2, 1e-22, lat.field(b0))
    xo = O.new_field()
    ito = O.cg("Hphi_sq", 0.2, 1e-22, xo, b0.copy())
    ito = ito[0] if isinstance(ito, tuple) else ito
    assert abs(it - ito) <= 1
    assert np.abs(x - xo)[:O.Vh].max() < 1e-7 * np.abs(xo[:O.Vh]).max()
