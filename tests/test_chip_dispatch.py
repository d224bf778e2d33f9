"""Which kernels run a case, and what the choice may change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _item(pkg, nx, ny, **kw):
    cfg = pkg.configs
    return cfg.channel_case(nx, ny, seed=nx, Re=150.0, scheme=pkg.SCHEME_QUICK, block=cfg.centred_block(2, 1, 0.3),
                            porosity=0.5, Da=1e-3, Cf=0.55, Ri=0.8, scalars=True, **kw)


def test_fast_results_do_not_depend_on_the_split(gpu):
    """FAST arithmetic, 102 x 102 (on chip in 7 CTAs or more) and 153 x 153 (in 16 only): every split that
    a caller asks for gives the same bits, iteration counts and errors, also those the case does not fit in."""
    for nx in (102, 153):
        prm, mesh, st, itc = _item(gpu, nx, nx, itc_max=25, arith=gpu.ARITH_FAST)
        ref = None
        for K in (0, 1, 4, 7, 16):
            b = gpu.Batch([prm], [mesh])
            b.set_cluster_size(0, K)
            b.set_state(0, st)
            _, it, er, _ = b.run(2, [itc])
            out = b.get_state(0)
            b.close()
            if ref is None:
                ref = (it, er, out)
            assert np.array_equal(it, ref[0]) and np.array_equal(er, ref[1]), K
            for k in out:
                assert np.array_equal(out[k], ref[2][k]), (K, k)


def test_the_choice_of_kernels(gpu):
    """What the library chooses by itself, and with ACS_OPT_ON_CHIP = 1."""
    small = _item(gpu, 30, 22, itc_max=4, arith=gpu.ARITH_FAST)
    art = gpu.configs.reference_case(12, itc_max=4, b_art=0.3)[:4]
    large = _item(gpu, 300, 300, itc_max=4, arith=gpu.ARITH_FAST)

    def used(item, n, engine, on_chip):
        b = gpu.Batch([item[0]] * n, [item[1]] * n)
        assert b.engines_used() == 0
        b.set_option(gpu.OPT_ENGINE, engine)
        b.set_option(gpu.OPT_ON_CHIP, on_chip)
        for c in range(n):
            b.set_state(c, item[2])
        b.run(1, item[3])
        r = b.engines_used()
        b.set_option(gpu.OPT_ON_CHIP, 1 - on_chip)  # takes effect with the next run
        b.run(1, item[3])
        assert r in (gpu.USED_CLUSTER, gpu.USED_GRAPH, gpu.USED_TILE, gpu.USED_CHIP)
        b.close()
        return r

    assert used(small, 3, gpu.ENGINE_CLUSTER, 0) == gpu.USED_CHIP
    assert used(small, 3, gpu.ENGINE_CLUSTER, 1) == gpu.USED_CLUSTER
    assert used(small, 3, gpu.ENGINE_TILE, 0) == gpu.USED_CHIP
    assert used(small, 3, gpu.ENGINE_TILE, 1) == gpu.USED_TILE
    assert used(small, 3, gpu.ENGINE_GRAPH, 0) == gpu.USED_GRAPH
    assert used(art, 1, gpu.ENGINE_CLUSTER, 0) == gpu.USED_CLUSTER
    assert used(large, 1, gpu.ENGINE_CLUSTER, 0) == gpu.USED_CLUSTER
    assert used(large, 1, gpu.ENGINE_TILE, 0) == gpu.USED_TILE
    c = gpu.Case(small[0], small[1])
    c.set_state(small[2])
    c.physical_steps(1, small[3])
    assert c.engines_used() == gpu.USED_CHIP
    for bad in (-1, 2):
        with pytest.raises(gpu.AcsError):
            c.set_option(gpu.OPT_ON_CHIP, bad)
    c.close()


@pytest.mark.parametrize("n,nx,ny,used", [(3, 40, 30, "USED_CHIP"), (1, 40, 30, "USED_CHIP"), (2, 300, 300, "USED_TILE")])
def test_loop_kind_does_not_choose_kernels(gpu, monkeypatch, n, nx, ny, used):
    """ACS_NO_CONDITIONAL_GRAPH sets how the loop of the graph and tile engines is driven; the kernels of a
    batch, and so its bits, stay."""
    item = _item(gpu, nx, ny, itc_max=12, arith=gpu.ARITH_FAST)
    outs = []
    for env in (False, True):
        if env:
            monkeypatch.setenv("ACS_NO_CONDITIONAL_GRAPH", "1")
        b = gpu.Batch([item[0]] * n, [item[1]] * n)
        b.set_option(gpu.OPT_ENGINE, gpu.ENGINE_TILE)
        for c in range(n):
            b.set_state(c, item[2])
        b.run(1, item[3])
        assert b.engines_used() == getattr(gpu, used)
        outs.append(b.get_state(n - 1))
        b.close()
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k]), k


def _ends(pkg):
    """Cases, a value put into one field, and runs: steps that end at itc_max, by the exit test (also in the
    first iterations), and with a residual that is NaN or infinite, from each field that can cause it."""
    cfg = pkg.configs
    full = dict(arith=pkg.ARITH_FAST)
    ref = lambda **kw: cfg.reference_case(12, arith=pkg.ARITH_FAST, **kw)[:4]  # noqa: E731
    plain = cfg.channel_case(45, 33, seed=4, Re=100.0, scheme=pkg.SCHEME_UPWIND, itc_max=40, arith=pkg.ARITH_FAST)
    capped = _item(pkg, 40, 30, itc_max=50, **full)
    return {
        "cap": (capped, None, [(2, 1), (1, 0)]),
        "exit": (_item(pkg, 30, 22, itc_max=3000, eps=3e-2, **full), None, [(3, 1), (2, 0)]),
        "exit-at-once": (_item(pkg, 30, 22, itc_max=3000, eps=1e3, **full), None, [(3, 1), (2, 0)]),
        "nan": (capped, ("um_tau", np.nan), [(3, 1)]),
        "overflow": (capped, ("vm", 1e150), [(3, 1)]),
        "T-inf": (capped, ("T", np.inf), [(3, 1)]),
        "C-nan": (capped, ("C_tau", np.nan), [(3, 1)]),
        "T-zero": (capped, ("T", 0.0), [(2, 1)]),
        "plain-cap": (plain, None, [(2, 1), (1, 0)]),
        "plain-p-inf": (plain, ("p", np.inf), [(2, 1)]),
        "plain-pn-nan": (plain, ("pn", np.nan), [(2, 1)]),
        "reference-cap": (ref(itc_max=40), None, [(2, 1), (1, 0)]),
        "reference-exit": (ref(itc_max=4000, eps=3e-3), None, [(4, 1), (2, 0)]),
        "reference-nan": (ref(itc_max=40), ("um", np.nan), [(2, 1)]),
    }


@pytest.mark.parametrize("engine", [0, 2], ids=["cluster", "tile"])
@pytest.mark.parametrize("end", ["cap", "exit", "exit-at-once", "nan", "overflow", "T-inf", "C-nan", "T-zero", "plain-cap",
                                 "plain-p-inf", "plain-pn-nan", "reference-cap", "reference-exit", "reference-nan"])
def test_on_chip_ends_like_the_engine_it_stands_in_for(gpu, engine, end):
    """FAST arithmetic, on chip and off: the same counts and status, every one of the 14 fields within 1e-10 of its
    largest value (the bound of the FAST engines) and with infinities and NaN at the same nodes, whatever
    ended the run."""
    from conftest import mask_dead
    (prm, mesh, st, itc), kick, runs = _ends(gpu)[end]
    st = {k: v.copy(order="F") for k, v in st.items()}
    if kick:
        st[kick[0]][5, 7] = kick[1]
    got = []
    for off in (0, 1):
        b = gpu.Batch([prm], [mesh])
        b.set_option(gpu.OPT_ENGINE, engine)
        b.set_option(gpu.OPT_ON_CHIP, off)
        b.set_state(0, st)
        log = [b.run(n, [i]) for n, i in runs]
        assert b.engines_used() == ((gpu.USED_TILE if engine else gpu.USED_CLUSTER) if off else gpu.USED_CHIP)
        got.append((log, b.get_state(0)))
        b.close()
    for x, y in zip(got[0][0], got[1][0]):
        for k in (0, 1, 3):
            assert np.array_equal(x[k], y[k])
        assert np.allclose(x[2], y[2], rtol=1e-9, atol=0.0, equal_nan=True)
    for k in got[0][1]:
        x, y = (mask_dead(k, g[1][k], prm.bc) for g in got)
        ok = np.isfinite(y)
        assert np.array_equal(np.isfinite(x), ok), k
        assert not ok.any() or np.abs(x[ok] - y[ok]).max() <= 1e-10 * np.abs(y[ok]).max(), k
