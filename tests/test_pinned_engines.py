"""The tile engine and the cluster engine on the cases that would run on chip by themselves.

The library sends small cases on these engines to the on-chip kernels, so the tests that name an engine
mostly run those.  Here the same tests run with ACS_OPT_ON_CHIP = 1, through a package whose batches and
cases set that option and check after every run which kernels it used."""
import pytest

import test_gpu_parity as parity
import test_long_horizon as horizon
import test_tile_engine as tile

pytestmark = pytest.mark.gpu


class _Pinned:
    """The package with batches and cases that never run on chip (`options`: further options of theirs)."""

    def __init__(self, pkg, options=()):
        self._pkg = pkg
        self.runs = 0
        outer = self
        expect = {pkg.ENGINE_CLUSTER: pkg.USED_CLUSTER, pkg.ENGINE_GRAPH: pkg.USED_GRAPH, pkg.ENGINE_TILE: pkg.USED_TILE}

        class Mixin:
            def __init__(self, *a):
                super().__init__(*a)
                self._engine = pkg.ENGINE_CLUSTER
                super().set_option(pkg.OPT_ON_CHIP, 1)
                for k, v in options:
                    super().set_option(k, v)

            def set_option(self, option, value):
                if option == pkg.OPT_ENGINE:
                    self._engine = value
                if option not in dict(options):
                    super().set_option(option, value)

            def _ran(self):
                assert self.engines_used() == expect[self._engine]
                outer.runs += 1

        class Batch(Mixin, pkg.Batch):
            def run(self, *a):
                r = super().run(*a)
                self._ran()
                return r

        class Case(Mixin, pkg.Case):
            def physical_steps(self, *a):
                r = super().physical_steps(*a)
                self._ran()
                return r

        self.Batch, self.Case = Batch, Case

    def __getattr__(self, name):
        return getattr(self._pkg, name)


@pytest.fixture
def pinned(gpu):
    p = _Pinned(gpu)
    yield p
    assert p.runs > 0


# ---- tile engine, conditional graph and overlapped launches -------------------------------------
@pytest.mark.parametrize("test", [tile.test_tile_engine_reference_case, tile.test_tile_engine_channel_full_physics,
                                  tile.test_tile_engine_ragged_batch], ids=lambda t: t.__name__[17:])
def test_tile_kernels(pinned, orc, test):
    test(pinned, orc)


@pytest.mark.parametrize("geom", tile.GEOMETRIES, ids=[f"{a}x{b}" for a, b in tile.GEOMETRIES])
def test_tile_kernels_geometries(pinned, orc, geom):
    tile.test_tile_engine_geometries(pinned, orc, geom)


@pytest.mark.parametrize("imax", [23, 40])
def test_tile_kernels_reference_variant_sizes(pinned, orc, imax):
    tile.test_tile_engine_reference_variant_sizes(pinned, orc, imax)


def test_tile_kernels_equal_graph_engine_fast(pinned):
    tile.test_tile_engine_equals_graph_engine_fast(pinned)


def test_tile_kernels_upload_between_steps_changes_nothing(pinned):
    tile.test_tile_engine_upload_between_steps_changes_nothing(pinned)


def test_tile_kernels_cfg1_200_steps(pinned):
    horizon.test_cfg1_200_steps_against_oracle(pinned, 2, 1)


def test_tile_kernels_host_polled_loop(pinned, orc, monkeypatch):
    """The loop that profilers can look into: one graph launch per pseudo-iteration."""
    monkeypatch.setenv("ACS_NO_CONDITIONAL_GRAPH", "1")
    tile.test_tile_engine_geometries(pinned, orc, (70, 33))


# ---- cluster engine ------------------------------------------------------------------------------
@pytest.mark.parametrize("test", [parity.test_loop_reference_small, parity.test_loop_channel_plain,
                                  parity.test_loop_channel_full_physics, parity.test_per_case_tolerance_bit_exact,
                                  parity.test_batch_equals_oracle_per_case], ids=lambda t: t.__name__[5:])
def test_cluster_kernels_exact(pinned, orc, test):
    test(pinned, orc, 0)


@pytest.mark.parametrize("nodes", [64, 300, 100000])
def test_cluster_kernels_splits(pinned, orc, nodes):
    parity.test_cluster_sizes_bit_exact(pinned, orc, nodes)


def test_cluster_kernels_per_case_splits(pinned):
    parity.test_per_case_cluster_sizes_bit_exact(pinned)


def test_cluster_kernels_failed_case(pinned):
    parity.test_failed_case_is_isolated(pinned)


# the FAST kernels: staged in shared memory, and from L2 and from L1 with one and two CTAs per SM
@pytest.mark.parametrize("staged,threads,per_sm,l1,long", [
    (1, 512, 1, 1, True), (1, 256, 1, 1, False), (0, 512, 1, 0, False), (0, 512, 1, 1, True),
    (0, 256, 1, 0, False), (0, 256, 1, 1, False), (0, 256, 2, 0, False), (0, 256, 2, 1, False)])
def test_cluster_kernels_fast(gpu, orc, staged, threads, per_sm, l1, long):
    """Converged steps of the reference case; `long`: of the full equation set too."""
    p = _Pinned(gpu, ((gpu.OPT_STAGED, staged), (gpu.OPT_THREADS, threads), (gpu.OPT_CTAS_PER_SM, per_sm)))
    parity.test_fast_engine_reference_case(p, orc, l1)
    if long:
        parity.test_fast_engine_channel_full_physics(p, orc, l1)
    assert p.runs == 1 + long
