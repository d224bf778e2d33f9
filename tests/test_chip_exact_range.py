"""EXACT arithmetic of the on-chip engine at the limits of its fast quotients: operands below 2^-900 (down to
subnormal numbers and zeros of both signs) and large ones, where it takes plain divisions, against the graph
engine's plain divisions, bit for bit."""
import numpy as np
import pytest

from conftest import mask_dead

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", ["full", "plain", "reference"])
@pytest.mark.parametrize("size", [1e-315, 1e-300, 1e-290, 1e-272, 1e-200, 1e60, 1e110, 1e150])
def test_extreme_states(gpu, flow, size):
    cfg = gpu.configs
    if flow == "reference":
        prm, mesh = cfg.reference_case(12, itc_max=4)[:2]
    else:
        kw = dict(scheme=gpu.SCHEME_QUICK, block=cfg.centred_block(2, 1, 0.3), porosity=0.4, Da=1e-3, Cf=0.55, Ri=1.0,
                  scalars=True) if flow == "full" else dict(scheme=gpu.SCHEME_UPWIND)
        prm, mesh, _, _ = cfg.channel_case(30, 22, itc_max=4, **kw)
    rng = np.random.default_rng(1)
    st = gpu.configs.zero_state(prm.imax, prm.jmax)
    for k, a in st.items():
        if k[0] == "T":
            a[:] = rng.uniform(0.5, 1.5, a.shape)
        else:  # magnitudes around `size`, some ordinary ones, some zeros
            a[:] = rng.choice([-1.0, 1.0], a.shape) * size * 10.0 ** rng.uniform(-6, 6, a.shape)
            pick = rng.uniform(0, 1, a.shape)
            a[pick < 0.1] = 0.0
            a[pick < 0.05] = -0.0
            a[pick > 0.9] = rng.uniform(-1e-2, 1e-2, int((pick > 0.9).sum()))
    got = []
    for engine in (gpu.ENGINE_CLUSTER, gpu.ENGINE_GRAPH):
        b = gpu.Batch([prm], [mesh])
        b.set_option(gpu.OPT_ENGINE, engine)
        b.set_state(0, st)
        r = b.run(2, [1])
        assert b.engines_used() == (gpu.USED_CHIP if engine == gpu.ENGINE_CLUSTER else gpu.USED_GRAPH)
        got.append((r, b.get_state(0)))
        b.close()
    for x, y in zip(got[0][0], got[1][0]):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
    for k in ("um", "vm", "p", "pn", "um_tau", "vm_tau", "um_n_tau", "vm_n_tau", "T", "C", "T_tau", "C_tau"):
        x, y = (mask_dead(k, g[1][k], prm.bc) for g in got)
        assert np.array_equal(x, y, equal_nan=True), (k, size)


@pytest.mark.parametrize("Re,Da,phi,Sc", [(1e-12, 1e-3, 0.4, 1.0), (1e15, 1e-3, 0.4, 1.0), (100.0, 1e-14, 0.4, 1.0), (100.0, 1e9, 0.4, 1.0),
                                          (100.0, 1e-3, 1e-12, 1.0), (100.0, 1e-3, 3.0, 1.0), (100.0, 1e-3, 0.4, 1e-13),
                                          (3.0, 1e-3, 1.0 / 3.0, 1.0), (0.1, 0.7, 0.1, 0.3)])
def test_extreme_constants(gpu, Re, Da, phi, Sc):
    """Divisors near the limits that the engine accepts, and ones whose reciprocals are not exact."""
    from dataclasses import replace
    cfg = gpu.configs
    prm, mesh, st, itc = cfg.channel_case(30, 22, seed=2, Re=Re, scheme=gpu.SCHEME_QUICK, block=cfg.centred_block(2, 1, 0.3),
                                          porosity=phi, Da=Da, Cf=0.55, Ri=1.0, scalars=True, itc_max=5)
    prm = replace(prm, Sc=Sc)
    got = []
    for engine in (gpu.ENGINE_CLUSTER, gpu.ENGINE_GRAPH):
        b = gpu.Batch([prm], [mesh])
        b.set_option(gpu.OPT_ENGINE, engine)
        b.set_state(0, st)
        r = b.run(2, [1])
        assert b.engines_used() == (gpu.USED_CHIP if engine == gpu.ENGINE_CLUSTER else gpu.USED_GRAPH)
        got.append((r, b.get_state(0)))
        b.close()
    for x, y in zip(got[0][0], got[1][0]):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
    for k in ("um", "vm", "p", "pn", "um_tau", "vm_tau", "um_n_tau", "vm_n_tau", "T", "C", "T_tau", "C_tau"):
        assert np.array_equal(got[0][1][k], got[1][1][k], equal_nan=True), k
