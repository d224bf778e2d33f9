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
