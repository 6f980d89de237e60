"""Kernels of whole runs that the device cannot schedule: the network runs on
the next form, ends on the launch plan as with engine="grid", and keeps no
array of the forms it left. Errors of the compiler are raised."""
import numpy as np
import pytest

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.core.backend import CompiledNetwork
from annarchy_b200.runtime.lib import BackendError, DryNative


class Native(DryNative):
    """Schedules clusters of up to `most` CTAs and `ctas` cooperative ones."""
    most, ctas, compiles = 0, 0, True

    def load_module(self, source, options):
        if not self.compiles:
            raise BackendError("anb_module_load", 3, "error")
        super().load_module(source, options)
        self.launches = None

    def set_local_kernel(self, name, grid, block, smem, cluster=1):
        if cluster == -1:
            self.local_grid = self.ctas
        elif cluster > self.most:
            raise BackendError("anb_set_local_kernel_ex", 1, "cannot be scheduled")

    def get_time(self):
        return 0


def _build(kind, engine="auto", **attrs):
    net = ann.Network(dt=1.0 if kind == "rate" else 0.1, seed=0)
    net.config(precision="double", engine=engine)
    rng = np.random.default_rng(1)
    n = 900 if kind == "rate" else 300
    if kind == "rate":
        pop = net.create(n, ann.Neuron(parameters="tau = 10.0 : population", equations="tau * dr/dt + r = sum(exc)"))
    else:
        pop = net.create(n, wl.coba_neuron(dict(wl.COBA_PARAMS)))
    w = wl.bernoulli_csr_skip(rng, n, n, 0.1, 0.1)
    net.connect(pop, pop, "exc").from_sparse(wl.to_from_sparse(w), 0.5 if kind == "delays" else 0.0)
    be = CompiledNetwork(net, dry=True)
    be.native = type("N", (Native,), attrs)()
    be.build()
    return be


@pytest.mark.parametrize("kind,attrs", [
    ("rate", dict(most=0, ctas=147)), ("rate", dict(most=8, ctas=0)), ("delays", dict(most=0))])
def test_what_cannot_be_scheduled_runs_on_the_plan(kind, attrs):
    be, plan = _build(kind, **attrs), _build(kind, "grid")
    assert be.engine == plan.engine == "grid" and be.masks is None
    source, same = (x.module.source.split("\n", 1)[1] for x in (be, plan))    # (without the network's number)
    assert source == same
    assert [x[0] for x in be.native.launches] == [x[0] for x in plan.native.launches]
    assert set(be.native.arrays) == set(plan.native.arrays)


@pytest.mark.parametrize("kind,attrs,kernel", [
    ("rate", dict(most=16, ctas=148), "anb_rate_run"), ("delays", dict(most=4), "anb_cluster_run"),
    ("plain", dict(most=4), "anb_cluster_run")])
def test_what_can_be_scheduled_stays(kind, attrs, kernel):
    be = _build(kind, **attrs)
    assert be.module.kernels == [kernel]
    assert be.engine == {"rate": "resident", "delays": "grid", "plain": "cluster"}[kind]


@pytest.mark.parametrize("kind", ["rate", "delays", "plain"])
def test_compiler_errors_are_raised(kind):
    with pytest.raises((BackendError, RuntimeError)):
        _build(kind, most=16, ctas=148, compiles=False)
