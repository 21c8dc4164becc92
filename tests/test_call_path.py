"""The host side of a kernel call: what it refuses before anything is launched, and its cached arguments."""

import pytest
import torch


@pytest.mark.parametrize("device", [torch.device("cpu"), "cpu", torch.device("meta")])
def test_no_stream_for_a_device_that_is_not_cuda(device):
    from voxneus_b200._lib import stream_ptr

    with pytest.raises(ValueError, match="Expected a cuda device"):
        stream_ptr(device)


def test_mlp_modules_refuse_host_tensors():
    """The MLP takes its device from its inputs: on host tensors it raises before any launch."""
    from voxneus_b200 import ops
    from voxneus_b200.models import RadianceMLP

    mlp = RadianceMLP()
    with pytest.raises((ValueError, RuntimeError)):
        mlp(torch.rand(5, 32), torch.rand(5, 16), torch.rand(5, 3))
    ws = [p.detach() for p in (mlp.net[0].weight, mlp.net[0].bias, mlp.net[2].weight, mlp.net[2].bias)]
    with pytest.raises(ValueError, match="Expected a cuda device"):
        ops.mlp_forward(torch.rand(5, 52), *ws)


def test_host_triples_keep_the_sign_of_zero():
    import math

    from voxneus_b200._lib import f3

    for v in ((0.0, 1.0, 2.0), (-0.0, 1.0, 2.0), (0.0, 1.0, 2.0)):
        assert math.copysign(1.0, f3(v)[0]) == math.copysign(1.0, v[0])
    assert f3((1, 2.5, -3))[:] == [1.0, 2.5, -3.0]
