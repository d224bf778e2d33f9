"""Field transfers: uploads and warm-start hooks that a caller captures into a CUDA graph, and transfers
of more than the staging buffer holds (2^23 doubles)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(pkg, nx=30, ny=22, **kw):
    cfg = pkg.configs
    return cfg.channel_case(nx, ny, seed=1, Re=150.0, scheme=pkg.SCHEME_QUICK, block=cfg.centred_block(2, 1, 0.3),
                            porosity=0.5, Da=1e-3, Cf=0.55, Ri=0.8, scalars=True, itc_max=20, **kw)


def _pinned(shape, value):
    import torch
    t = torch.full(shape[::-1], value, dtype=torch.float64).pin_memory()
    return t, t.numpy().T  # Fortran order


@pytest.mark.parametrize("when", ["fresh", "warm", "stream-in-capture"])
def test_captured_uploads(gpu, when):
    """Uploads from pinned memory captured into a graph, on a batch that has moved no field yet, on one
    that has, and with the stream handed over inside the capture.  Every replay takes what the host array
    holds then, also after later transfers of more fields than the capture saw."""
    import torch
    prm, mesh, st, itc = _case(gpu)
    b = gpu.Batch([prm], [mesh])
    if when != "fresh":
        b.set_state(0, {"vm": st["vm"]})
    s = torch.cuda.Stream()
    if when != "stream-in-capture":
        b.set_stream(s.cuda_stream)
    host, arr = _pinned(gpu.field_shape("um", 30, 22), 3.0)
    host2, arr2 = _pinned(gpu.field_shape("pn", 30, 22), 4.0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        if when == "stream-in-capture":
            b.set_stream(s.cuda_stream)
        b.set_state(0, {"um": arr, "pn": arr2})
    for value in (3.0, 5.0):
        host.fill_(value)
        g.replay()
        torch.cuda.synchronize()
        got = b.get_state(0)  # all fields: the staging buffer grows
        assert (got["um"] == value).all() and (got["pn"] == 4.0).all()
        b.set_state(0, st)
    b.close()


def test_captured_hook_after_an_upload(gpu):
    """An upload changes the control words (pn gets a buffer of its own again); warm-start features that
    are captured next leave them right for work outside the graph, before any replay."""
    import torch
    prm, mesh, st, itc = _case(gpu)
    pn = np.asfortranarray(np.random.default_rng(3).uniform(-1, 1, gpu.field_shape("pn", 30, 22)))
    X = torch.zeros(32 * 32 * 11, device="cuda")
    sc = torch.zeros(8, device="cuda")
    outs = []
    for captured in (False, True):
        s = torch.cuda.Stream()
        b = gpu.Batch([prm], [mesh])
        b.set_stream(s.cuda_stream)
        b.ws_enable(32, 32)
        b.set_state(0, st)
        b.run(1, [itc])
        b.set_state(0, {"pn": pn})
        g = torch.cuda.CUDAGraph()
        if captured:
            with torch.cuda.graph(g, stream=s):
                b.ws_features(X.data_ptr(), sc.data_ptr())
        b.ws_enable(32, 32)
        b.ws_features(X.data_ptr(), sc.data_ptr())
        torch.cuda.synchronize()
        outs.append(X.clone().cpu().numpy())
        b.close()
    canvas = outs[0].reshape(32, 32, 11)[:22, :30, 2]
    assert np.array_equal(canvas, pn.T.astype(np.float32))
    assert np.array_equal(outs[0], outs[1])


def _random_state(pkg, nx, ny, names):
    rng = np.random.default_rng(nx)
    return {k: np.asfortranarray(rng.uniform(0.5, 1.5, pkg.field_shape(k, nx, ny))) for k in names}


# 1999 x 1500: two fields fit in the staging buffer; 3003 x 2900: none does; 2890 x 2902: p fits, vm does not
@pytest.mark.parametrize("nx,ny", [(1999, 1500), (3003, 2900), (2890, 2902)])
def test_large_fields_keep_little_memory(gpu, nx, ny):
    """Fields come back as they were sent, and the device memory that transfers keep is bounded (64 MiB
    and what the allocator rounds it up to), however large the case."""
    import torch
    prm, mesh, st, itc = gpu.configs.channel_case(nx, ny, seed=1)
    del st
    names = ("um", "vm", "p", "pn", "T", "um_n_tau")
    st = _random_state(gpu, nx, ny, names)
    for make in (gpu.Case, gpu.Batch):
        b = gpu.Case(prm, mesh) if make is gpu.Case else gpu.Batch([prm], [mesh])
        args = () if make is gpu.Case else (0,)
        free = torch.cuda.mem_get_info()[0]
        b.set_state(*args, st)
        got = b.get_state(*args, names)
        assert free - torch.cuda.mem_get_info()[0] <= 80 << 20
        for k in names:
            assert np.array_equal(got[k], st[k]), k
        b.close()


def test_large_routine_calls(gpu, orc):
    """solve_P and solve_U of a case whose fields do not fit in the staging buffer, against the oracle."""
    nx, ny = 3003, 2900
    prm, mesh, _, _ = gpu.configs.channel_case(nx, ny, seed=1, scheme=gpu.SCHEME_UPWIND)
    a = _random_state(gpu, nx, ny, ("um", "um_tau", "vm_tau", "um_n_tau", "vm_n_tau", "p", "pn"))
    b = {k: v.copy(order="F") for k, v in a.items()}
    g, o = gpu.Case(prm, mesh), orc.OracleCase(prm, mesh)
    assert g.solve_P(a["p"], a["um_n_tau"], a["vm_n_tau"], a["pn"]) == o.solve_p(b["p"], b["um_n_tau"], b["vm_n_tau"], b["pn"])
    assert (g.solve_U(a["um"], None, None, a["um_tau"], a["vm_tau"], a["um_n_tau"], a["pn"])
            == o.solve_u(b["um"], b["um_tau"], b["vm_tau"], b["pn"], b["um_n_tau"]))
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    g.close()


@pytest.mark.parametrize("nx,ny", [(51, 20), (52, 21), (50, 9), (6, 6)])
@pytest.mark.parametrize("pin", [False, True])
def test_routes_of_small_fields(gpu, nx, ny, pin):
    """Fields with and without padding between their rows (um of 51 x 20, vm of 52 x 21 have none), one
    at a time and together, pageable and pinned, mixed in one call: each comes back as it was sent."""
    prm, mesh, _, _ = gpu.configs.channel_case(nx, ny, seed=1)
    st = _random_state(gpu, nx, ny, gpu.FIELDS)
    if pin:
        st = {k: (_pinned(a.shape, 0.0)[1], a) for k, a in st.items()}
        for v, a in st.values():
            v[:] = a
        st = {k: v for k, (v, a) in st.items()}
    b, c = gpu.Batch([prm], [mesh]), gpu.Case(prm, mesh)
    b.set_state(0, st)
    c.set_state(st)
    for got in (b.get_state(0), c.get_state(), {k: b.get_state(0, (k,))[k] for k in st}):
        for k in st:
            assert np.array_equal(got[k], st[k]), k
    out = {k: _pinned(a.shape, -1.0)[1] if pin else np.full_like(a, -1.0) for k, a in st.items()}
    for k in st:
        b.get_state(0, (k,), out=out)
        assert np.array_equal(out[k], st[k]), k
    b.close()
    c.close()
