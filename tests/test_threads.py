"""Two host threads that use the library at once, each with objects of its own: launches of one kernel
with different amounts of shared memory must not get into each other's way."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _run(jobs):
    errors = []
    start = threading.Barrier(len(jobs))

    def go(job):
        try:
            start.wait()
            job()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=go, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("kernel", ["conv3x3", "gather", "dx"])
def test_network_kernels_of_different_sizes(gpu, kernel):
    """The same kernel instance for few and for many channels, each thread on its own stream."""
    import importlib
    import torch
    L = importlib.import_module("solver_cfd_b200.unet").kernels()
    B, H, W, Cout = 1, 16, 16, 32

    def job(Cc, n):
        s = torch.cuda.Stream()
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        with torch.cuda.stream(s):
            if kernel == "dx":
                dz = torch.randn(B * H * W, Cc, device="cuda").to(torch.bfloat16)
                wt = torch.randn(9 * Cout, Cc, device="cuda").to(torch.bfloat16)
                y = torch.zeros(B * H * W, Cout, device="cuda")
            else:
                x = torch.randn(B * H * W, Cc, device="cuda").to(torch.bfloat16)
                kp = (9 * Cc + 7) // 8 * 8
                wt = torch.randn(Cout, kp, device="cuda").to(torch.bfloat16)
                y = torch.zeros(B * H * W, Cout, device="cuda", dtype=torch.bfloat16)
        s.synchronize()

        def go():
            for _ in range(n):
                if kernel == "dx":
                    r = L.unet_conv3x3_dx(dz.data_ptr(), wt.data_ptr(), B, H, W, Cout, Cc, y.data_ptr(), err.data_ptr(),
                                          s.cuda_stream)
                elif kernel == "gather":
                    r = L.unet_conv3x3_gather(x.data_ptr(), B, H, W, Cc, wt.data_ptr(), kp, kp, Cout, y.data_ptr(), Cout,
                                              None, 0, err.data_ptr(), s.cuda_stream)
                else:
                    r = L.unet_conv3x3(x.data_ptr(), B, H, W, Cc, wt.data_ptr(), kp, Cout, 2, None, y.data_ptr(), Cout,
                                       None, 0, err.data_ptr(), s.cuda_stream)
                assert r == 0, r
            s.synchronize()
            assert int(err.item()) == 0
        return go

    _run([job(3 if kernel == "gather" else 16, 20000), job(11 if kernel == "gather" else 256, 20000)])


@pytest.mark.parametrize("arith", [0, 1], ids=["exact", "fast"])
def test_batches_of_different_sizes(gpu, arith):
    """Batches of small and of larger cases, a few pseudo-iterations per run."""
    cfg = gpu.configs

    def job(nx, ny, n):
        prm, mesh, st, itc = cfg.channel_case(nx, ny, seed=1, Re=150.0, scheme=gpu.SCHEME_QUICK,
                                              block=cfg.centred_block(2, 1, 0.3), porosity=0.5, Da=1e-3, Cf=0.55,
                                              Ri=0.8, scalars=True, itc_max=3, arith=arith)
        b = gpu.Batch([prm], [mesh])
        b.set_state(0, st)

        def go():
            for _ in range(n):
                b.run(1, [itc])
        return go

    _run([job(20, 26, 3000), job(60, 62, 3000), job(30, 40, 3000)])
