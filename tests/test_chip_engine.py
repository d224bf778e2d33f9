"""The on-chip engine (whole pseudo-time state in a cluster's shared memory, EXACT arithmetic) against
the CPU oracle, bit for bit, from states that do not satisfy the boundary passes: both boundary
variants, both schemes, with and without scalars, every cluster size a case allows, strips of the
smallest height, physical-step arrays on and off the chip, steps that end at itc_max and by
convergence, runs that continue a state, and cases that the engine leaves to the cluster engine."""
import numpy as np
import pytest

from conftest import fcopy, mask_dead

pytestmark = pytest.mark.gpu

# (nx, ny, clusters): 6 x 6 is the smallest case; 7 x 33 and 40 x 9 the thinnest strips; 153 x 60 in 7
# CTAs keeps its physical-step arrays in global memory; 290 x 40 is wider than a CTA has threads
SIZES = [(6, 6, (1,)), (7, 33, (1, 3, 8)), (40, 9, (2,)), (35, 63, (1, 5, 16)), (153, 60, (7, 15)), (290, 40, (10,))]


def _state(pkg, nx, ny, seed):
    rng = np.random.default_rng(seed)
    st = pkg.configs.zero_state(nx, ny)
    for k, a in st.items():
        lo, hi = (0.5, 1.5) if k[0] == "T" else (0.0, 1.0) if k[0] == "C" else (-1e-2, 1e-2)
        a[:] = rng.uniform(lo, hi, a.shape)
    return st


def _case(pkg, flow, nx, ny, **kw):
    cfg = pkg.configs
    if flow == "reference":
        prm, mesh, _, _, _ = cfg.reference_case(nx, **kw)
        return prm, mesh
    full = flow == "full"
    prm, mesh, _, _ = cfg.channel_case(nx, ny, scheme=pkg.SCHEME_QUICK if full else pkg.SCHEME_UPWIND,
                                       block=cfg.centred_block(2, 1, 0.3) if full else None,
                                       porosity=0.4 if full else 1.0, Da=1e-3, Cf=0.55, Ri=1.0, scalars=full,
                                       T_block=2.0, **kw)
    return prm, mesh


def _compare(pkg, orc, prm, mesh, clusters, runs, seed=3):
    """runs: [(physical steps, itc)], each continuing the state of the one before."""
    st = _state(pkg, prm.imax, prm.jmax, seed)
    for K in clusters:
        b = pkg.Batch([prm], [mesh])
        if K:
            b.set_cluster_size(0, K)
        b.set_state(0, st)
        o, ost = orc.OracleCase(prm, mesh), fcopy(st)
        for steps, itc in runs:
            itc_g, it_g, er_g, _ = b.run(steps, itc)
            itc_o, it_o, er_o = o.run(ost, steps, itc)
            assert list(it_g[0]) == list(it_o) and itc_g[0] == itc_o and np.array_equal(er_g[0], er_o), (K, er_g, er_o)
            out = b.get_state(0)
            for k in out:
                if prm.solve_scalars or k[0] not in "TC":
                    x, y = mask_dead(k, out[k], prm.bc), mask_dead(k, ost[k], prm.bc)
                    assert np.array_equal(x, y), (K, k, float(np.nanmax(np.abs(x - y))))
        b.close()


@pytest.mark.parametrize("flow", ["full", "plain"])
@pytest.mark.parametrize("nx,ny,clusters", SIZES, ids=[f"{a}x{b}" for a, b, _ in SIZES])
def test_channel_sizes(gpu, orc, flow, nx, ny, clusters):
    prm, mesh = _case(gpu, flow, nx, ny, itc_max=4)
    _compare(gpu, orc, prm, mesh, clusters, [(2, 1), (1, 0)])


@pytest.mark.parametrize("imax", [6, 12, 25])
@pytest.mark.parametrize("scheme", [0, 1])
def test_reference_variant(gpu, orc, imax, scheme):
    prm, mesh = _case(gpu, "reference", imax, 0, itc_max=5, scheme=scheme)
    _compare(gpu, orc, prm, mesh, (1, 2, 0), [(2, 1), (1, 0)])


def test_steps_that_converge(gpu, orc):
    """Loose tolerance: steps end by the exit test, some in the first pseudo-iterations."""
    for flow, nx, ny in (("full", 30, 22), ("reference", 12, 0)):
        prm, mesh = _case(gpu, flow, nx, ny, itc_max=3000, eps=3e-2 if flow == "full" else 3e-3)
        _compare(gpu, orc, prm, mesh, (0, 2), [(4, 1), (3, 0)])


def test_cases_left_to_the_cluster_engine(gpu, orc):
    """Damping, and a case larger than a cluster's shared memory."""
    prm, mesh = _case(gpu, "reference", 12, 0, itc_max=4, b_art=0.3)
    _compare(gpu, orc, prm, mesh, (0,), [(2, 1)])
    prm, mesh = _case(gpu, "full", 210, 205, itc_max=3)
    _compare(gpu, orc, prm, mesh, (0,), [(1, 1)])


@pytest.mark.parametrize("nx,ny", [(61, 45), (70, 33), (20, 26)])
def test_tile_kernels_on_small_cases(gpu, orc, monkeypatch, nx, ny):
    """Small batches on the tile engine run on chip; with the host-polled loop they stay on the tile
    kernels.  Both against the oracle at the FAST arithmetic's bound (1e-10)."""
    from test_tile_engine import _tile_vs_oracle
    item = gpu.configs.channel_case(nx, ny, seed=nx, Re=150.0, scheme=gpu.SCHEME_QUICK,
                                    block=gpu.configs.centred_block(2, 1, 0.3), porosity=0.5, Da=1e-3, Cf=0.55, Ri=0.8,
                                    scalars=True, itc_max=100)
    _tile_vs_oracle(gpu, orc, [item], 2)
    monkeypatch.setenv("ACS_NO_CONDITIONAL_GRAPH", "1")
    _tile_vs_oracle(gpu, orc, [item], 2)
