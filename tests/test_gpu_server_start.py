"""A query submitted the moment a server exists: its command must not be wiped by
the server's own resets, which take longest with many slots and large rings."""
import time

import numpy as np
import pytest

import oracle_lib
from mlmq_tpds_withl3_b200 import DeviceGraph, HostGraph
from mlmq_tpds_withl3_b200.server import Server

pytestmark = pytest.mark.gpu


def test_queries_submitted_at_once_are_served():
    import torch
    g = HostGraph.grid(64, 64, seed=71)
    dg = DeviceGraph.upload(g)
    ref, _ = oracle_lib.sssp_i32(g, 3)
    bufs = [torch.empty(g.n, dtype=torch.int32, pin_memory=True) for _ in range(64)]
    for _ in range(2):  # the second server takes pooled memory and starts sooner
        sv = Server(64, g.n, {"l2_cap_log2": 19}, lifetime_s=5.0)
        tickets = [sv.submit(dg, 3, b) for b in bufs]
        assert None not in tickets
        done, t0 = {}, time.time()
        while len(done) < len(tickets) and time.time() - t0 < 10:
            done.update(dict(sv.poll()))
        sv.close()
        assert done == {t: 0 for t in tickets}
        for b in bufs:
            assert np.array_equal(b.numpy(), ref)
