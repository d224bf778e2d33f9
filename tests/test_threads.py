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
