"""Surrogate fields of networks of different shapes, evaluated by several threads at once."""

import threading

import numpy as np
import pytest
import torch

from pyftle_b200 import _lib
from pyftle_b200._device import ptr, stream_ptr
from pyftle_b200.surrogate import FlowMapMLP

pytestmark = pytest.mark.gpu


def _net(hidden, depth):
    rng = np.random.default_rng(hidden)
    freq = np.zeros((32, 4), dtype=np.float32)
    freq[:, :3] = np.round(rng.normal(0.0, 3.0, (32, 3)))
    return FlowMapMLP(freq, hidden=hidden, depth=depth, out_scale=0.05, seed=hidden)


def _field_call(net, points, out):
    """Arguments of the field kernel's entry point, its weights packed."""
    shape = (net.dim, net.hidden, net.depth, net.freq.shape[0])
    packed = torch.empty(_lib.load().ftle_mlp_field_bytes(*shape), dtype=torch.uint8,
                         device="cuda")
    _lib.call("ftle_mlp_field_pack", *shape, ptr(net.wb), ptr(packed), stream_ptr())
    args = (*shape, ptr(points), points.shape[0], ptr(packed), ptr(net.w), ptr(net.freq),
            net.out_scale, 5.0, ptr(out), ptr(net.err), stream_ptr())
    return args, packed


# shapes that share a kernel instance and differ in the shared memory they launch with
@pytest.mark.parametrize("shapes", [((192, 1), (384, 4)), ((64, 1), (128, 4))])
def test_threads_with_networks_of_different_sizes(shapes):
    points = torch.rand(8, 3, dtype=torch.float64, device="cuda")
    nets = [_net(*s) for s in shapes for _ in range(2)]
    outs = [torch.empty(8, dtype=torch.float64, device="cuda") for _ in nets]
    calls = [_field_call(net, points, out) for net, out in zip(nets, outs)]
    torch.cuda.synchronize()
    lib, errors, start = _lib.load(), [], threading.Barrier(len(nets))

    def work(args):
        start.wait()
        for _ in range(5000):
            if lib.ftle_mlp_field(*args) != 0:  # the host's status of the launch
                errors.append(lib.ftle_last_error())
                return

    threads = [threading.Thread(target=work, args=(args,)) for args, _ in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert errors == []
    for net, out in zip(nets, outs):
        assert torch.equal(out, net.ftle(points, 5.0))
