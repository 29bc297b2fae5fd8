"""A call that fails after it has enqueued work returns with its stream idle: its constants go out of, and its flags
come back to, a pinned block that the next call writes."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


def test_failed_walk_leaves_nothing_in_flight(cuda_lib):
    import torch

    ic = ics.grid_box(n1=12, seed=2, pmgrid=24)
    n = len(ic["mass"])
    old = np.full(n, 0.3, np.float32)
    ewald = L.make_params(True, softening=ic["softening"], precision=L.PREC_FP32, err_tol_theta=0.0)
    group64 = L.make_params(True, softening=ic["softening"], precision=L.PREC_FP64_GROUP, err_tol_theta=0.0)  # has no Ewald form
    stream = torch.cuda.Stream()
    a = torch.ones(8192, 8192, device="cuda")
    with GravityTree(ewald) as t:
        t.set_stream(stream.cuda_stream)
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        good = t.gravity_tree(old)
        t.set_params(group64)
        torch.cuda.synchronize()
        for _ in range(3):
            with torch.cuda.stream(stream):
                for _ in range(12):  # some 200 ms of work ahead of the call's own
                    b = a @ a
            with pytest.raises(L.GpuGravError):
                t.gravity_tree(old)
            assert stream.query()
        t.set_params(ewald)
        for x, y in zip(t.gravity_tree(old), good):
            assert np.array_equal(x, y)
        t.set_stream(None)
    del a, b
