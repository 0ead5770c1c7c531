"""Sweeps at the edges of their tiles, runs and layouts: lattices one site short of a tile, one site
over and ragged, against the FP64 oracle at the parity tests' bars (1e-12 of each component's
maximum), and the lphi4SU2U1 site orders against each other."""
import numpy as np
import pytest

from conftest import make_su2_case, make_u1_case

pytestmark = pytest.mark.gpu

TOL = 1e-12


def rel(a, b, nc):
    a, b = np.asarray(a).reshape(nc, -1), np.asarray(b).reshape(nc, -1)
    sc = np.abs(b).max(axis=1)
    return max(np.abs(a[c] - b[c]).max() / sc[c] if sc[c] > 0 else np.abs(a[c]).max() for c in range(nc))


@pytest.mark.parametrize("N", [7, 31, 33, 41])
@pytest.mark.parametrize("evolver", ["VV2", "LF"])
def test_gw_sweep_on_ragged_tiles(N, evolver):
    # tiles of 32 x 8 sites, runs of 4 planes and more; the first kick, drift-and-kick sweeps, the
    # last drift and the sync's half kick
    from cosmolattice_b200 import Lattice, ParameterParser, RunParameters, lphi4_1f
    from oracle.oracle import OracleLattice

    par = ParameterParser(params={"N": N, "kIR": 1.0, "dt": 0.005, "evolver": evolver, "expansion": "true", "lambda": 1.0,
                                  "initial_amplitudes": "5.6964e18"})
    rp = RunParameters(par)
    m = lphi4_1f(par, rp)
    rng = np.random.default_rng(N)
    f, p = 1.0 + 1e-2 * rng.standard_normal(N ** 3), 1e-2 * rng.standard_normal(N ** 3)
    u, pi = 1e-2 * rng.standard_normal(5 * N ** 3), 1e-2 * rng.standard_normal(5 * N ** 3)
    sf = {"aI": 1.0, "aSI": 1.0, "aIM": 1.0, "aDotI": 0.5, "aDotSI": 0.5}
    out = []
    for cls in (Lattice, OracleLattice):
        lat = cls(m, rp)
        lat.gws_enable()
        lat.set_state(f, p, sf)
        lat.gws_set_state(u, pi)
        lat.initialize()
        lat.evolve(5)
        lat.evolve(1)
        lat.sync()
        out.append(lat.gws_get_state())
        lat.close()
    for a, b in zip(*out):
        assert rel(a, b, 5) < TOL


@pytest.mark.parametrize("N", [5, 9, 33])
def test_su2_state_round_trip_and_step(N):
    # the device layout's padding (6 N^3 elements to a multiple of four): every component comes back as
    # it was set, and a step agrees with the oracle
    from cosmolattice_b200 import Lattice
    from oracle.oracle import OracleLattice

    par, rp, m, f, p, sf = make_su2_case(N=N, evolver="VV2", expansion=True, amp=3e-2)
    rng = np.random.default_rng(N)
    f = f + 1e-2 * rng.standard_normal(f.shape)
    for i in range(3):
        f[10 + 4 * i:14 + 4 * i] /= np.sqrt((f[10 + 4 * i:14 + 4 * i] ** 2).sum(axis=0))
    out = []
    for cls in (Lattice, OracleLattice):
        lat = cls(m, rp)
        lat.set_state(f, p, sf)
        if cls is Lattice:
            g = lat.get_state()
            assert np.array_equal(g[0].ravel(), f.ravel()) and np.array_equal(g[1].ravel(), p.ravel())
        lat.initialize()
        lat.evolve(3)
        out.append(lat.get_state())
        lat.close()
    assert rel(out[0][0], out[1][0], 22) < TOL and rel(out[0][1], out[1][1], 19) < TOL


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("fp32", 1e-6)])
def test_su2_site_orders_compute_the_same_step(monkeypatch, precision, tol):
    # linear and bricks (runs that do and do not divide N): the same sites, other groupings of the sums
    from cosmolattice_b200 import Lattice

    par, rp, m, f, p, sf = make_su2_case(N=35, evolver="VV2", expansion=True, amp=3e-2)
    res = []
    for order in ("0", "1", "3", "35", "64"):
        monkeypatch.setenv("CLB_GAUGE_ORDER", order)
        lat = Lattice(m, rp, precision=precision)
        lat.set_state(f, p, sf)
        lat.initialize()
        lat.evolve(4)
        res.append(lat.get_state())
        lat.close()
    for r in res[1:]:
        assert rel(r[0], res[0][0], 22) < tol and rel(r[1], res[0][1], 19) < tol


@pytest.mark.parametrize("tangent", [False, True])
@pytest.mark.parametrize("N,order", [(5, 0), (33, 0), (33, 1), (34, 5)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_su2_force_by_direction_is_the_whole_sweep(monkeypatch, precision, N, order, tangent):
    # the SU(2) part with a thread per site and direction against the one-thread sweep over every
    # sector, in lattices that end inside a block, a tile and a run: states and a(t) to the last bit
    from cosmolattice_b200 import Lattice
    from cosmolattice_b200.initializers import su2u1_initial_state_tangent

    monkeypatch.setenv("CLB_GAUGE_ORDER", str(order))
    par, rp, m, f, p, sf = make_su2_case(N=N, evolver="VV2", expansion=True, amp=3e-2)
    rng = np.random.default_rng(N)
    f = f + 1e-2 * rng.standard_normal(f.shape)
    for i in range(3):
        f[10 + 4 * i:14 + 4 * i] /= np.sqrt((f[10 + 4 * i:14 + 4 * i] ** 2).sum(axis=0))
    out = []
    for split in ("0", "3"):
        monkeypatch.setenv("CLB_SU2_SPLIT", split)
        lat = Lattice(m, rp, precision=precision)
        lat.set_state(f, p, sf)
        if tangent:
            df, dp, cd = su2u1_initial_state_tangent(m, rp, "gSU2", (f, p))
            lat.tangent_begin(cd, df, dp)
        lat.initialize()
        lat.evolve(3)
        out.append([lat.get_state()] + ([lat.tangent_get_state()] if tangent else []))
        lat.close()
    for a, b in zip(*out):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_su2_state_round_trip_in_several_runs_of_the_staging_buffer(precision):
    # 205^3 sites: a whole run of 2^23 and a remainder; every value is a whole number below 2^24, which
    # FP32 holds
    from cosmolattice_b200 import MODELS, Lattice, ParameterParser, RunParameters

    N = 205
    par = ParameterParser(params={"N": N, "kIR": 1.0, "dt": 0.005, "evolver": "VV2", "expansion": "true", "lambda": 1.0,
                                  "qG": 50.0, "qH": 50.0, "SU2Doublet_initial_norm": "5.25151e18", "gU1s": 0.35, "gSU2s": 0.6})
    rp = RunParameters(par)
    m = MODELS["lphi4SU2U1"](par, rp)
    base = np.arange(N ** 3, dtype=np.float64).reshape(N, N, N)
    f, p = np.empty((22, N, N, N)), np.empty((19, N, N, N))
    for c in range(22):
        f[c] = base + c
    for c in range(19):
        p[c] = base + 100 + c
    lat = Lattice(m, rp, precision=precision)
    lat.set_state(f, p, {"aI": 1.0, "aSI": 1.0, "aIM": 1.0, "aDotI": 0.0, "aDotSI": 0.0})
    g = lat.get_state()
    lat.close()
    assert np.array_equal(g[0].ravel(), f.ravel()) and np.array_equal(g[1].ravel(), p.ravel())


def test_su2_handle_holds_no_more_than_its_state_and_phases():
    # 22 fields, 19 momenta and 12 phases per site, a staging buffer of 64 MiB and small change (partial
    # sums, the allocator's granularity: under 32 MiB)
    import torch

    from cosmolattice_b200 import MODELS, Lattice, ParameterParser, RunParameters

    N = 256
    par = ParameterParser(params={"N": N, "kIR": 1.0, "dt": 0.005, "evolver": "VV2", "expansion": "true", "lambda": 1.0,
                                  "qG": 50.0, "qH": 50.0, "SU2Doublet_initial_norm": "5.25151e18", "gU1s": 0.35, "gSU2s": 0.6})
    rp = RunParameters(par)
    m = MODELS["lphi4SU2U1"](par, rp)
    Lattice(m, rp).close()  # the context and the kernels are loaded
    free = torch.cuda.mem_get_info()[0]
    lat = Lattice(m, rp)
    held = free - torch.cuda.mem_get_info()[0]
    lat.close()
    assert held <= 53 * 8 * N ** 3 + (96 << 20), held


@pytest.mark.parametrize("make", [make_u1_case, make_su2_case])
@pytest.mark.parametrize("evolver", ["VV2", "LF"])
def test_gauge_loops_without_dependent_launches(monkeypatch, make, evolver):
    # CLB_PDL=0 launches every kernel after the one before has drained: the same state to the last bit
    from cosmolattice_b200 import Lattice

    par, rp, m, f, p, sf = make(N=19, evolver=evolver, expansion=True, amp=3e-2)
    res = []
    for pdl in ("1", "0"):
        monkeypatch.setenv("CLB_PDL", pdl)
        lat = Lattice(m, rp)
        lat.set_state(f, p, sf)
        lat.initialize()
        lat.evolve(6)
        lat.sync()
        res.append(lat.get_state())
        lat.close()
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1]) and res[0][2] == res[1][2]
