"""The serving loop's binding fills its request table from columns (no device calls: runs without a
GPU)."""
import numpy as np
import pytest
import torch


def test_server_run_takes_columns_of_any_kind(pbm_mod):
    """Lists, arrays, float-valued counts and tensors fill the same requests; a short column is refused."""
    pbm = pbm_mod
    seen = []

    class Lib:
        def pbm_server_run(self, h, reqs, n, res, rep):
            seen.append([(r.arrival_s, r.tenant, r.op, r.count) for r in reqs])
            return 0

    srv = pbm.Server.__new__(pbm.Server)
    srv.lib, srv.h = Lib(), None
    want = [(0.0, 3, 0, 5), (0.5, 1, 1, 1 << 30), (2.0, 0, 2, 7)]
    cols = [list(c) for c in zip(*want)]
    srv.run(*cols)
    srv.run(*[tuple(c) for c in cols])
    srv.run(*[np.array(c) for c in cols])
    srv.run(*[torch.tensor(c) for c in cols])
    srv.run(cols[0], [3.0, 1.9, 0.2], cols[2], np.array(cols[3], dtype=np.uint32))
    srv.run(cols[0], [3 + (1 << 32), 1, 1 << 70], cols[2], cols[3])
    assert seen == [want] * 6
    srv.run([], [], [], [])
    assert seen[-1] == []
    with pytest.raises(IndexError):
        srv.run(cols[0], [3], cols[2], cols[3])
    with pytest.raises(ValueError):
        srv.run(cols[0], [float("nan"), 1.0, 2.0], cols[2], cols[3])
