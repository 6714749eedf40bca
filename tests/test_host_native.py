"""The native walk over a net's parameters (csrc/host.cpp)."""
import torch
import torch.nn as nn

import dlr_lock_b200 as D
from dlr_lock_b200.build import build_library


def test_any_change_of_a_parameter_is_seen():
    build_library()
    host = D._lib.host()
    net = D.DLRNet(32, 4, 3)
    dicts = net._param_dicts
    key = host.snapshot(dicts())
    assert len(key) == 16 * 12 and host.unchanged(key, dicts())
    with torch.no_grad():
        net.Us[2].mul_(2.0)                                    # in place
    assert not host.unchanged(key, dicts())
    key = host.snapshot(dicts())
    net.Vs[1].data = torch.zeros(4, 32)                        # another storage behind the same parameter
    assert not host.unchanged(key, dicts())
    key = host.snapshot(dicts())
    net.alphas[0] = nn.Parameter(torch.tensor(1.0))            # another parameter
    assert not host.unchanged(key, dicts())
    key = host.snapshot(dicts())
    net.rms_w.append(nn.Parameter(torch.ones(32)))             # one more
    assert not host.unchanged(key, dicts()) and host.unchanged(host.snapshot(dicts()), dicts())
    # parameters on the CPU are not for the fold kernel
    assert host.layers(dicts()) is None and host.state_layers(net.state_dict()) is None
