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
