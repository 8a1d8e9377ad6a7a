"""A batch's limit of 256-nonzero chunks: a matrix of more is refused, unless a
run of more than 256 empty rows has it served on its own; the statistics count
such chunks."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


def _matrix(run, rows):
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(5)
    lens = np.concatenate([np.full(rows // 2, 9), np.zeros(run, int), np.full(rows - rows // 2, 9)])
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return HostCSR(len(lens), 700, rp, rng.integers(0, 700, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1]))


def test_more_chunks_than_a_batch():
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300._lib import SSPMVError
    from sspmv_gb300.serving import Server
    mats = {0: _matrix(300, 1000), 1: _matrix(256, 1000), 2: _matrix(300, 200)}  # 36, 36 and 8 chunks
    x = np.random.default_rng(1).uniform(-1, 1, 700)
    with Server(max_batch_tiles=16) as s:
        for i, A in mats.items():
            s.add_matrix(i, A)
        for i in (0, 2):
            y = np.empty(mats[i].num_rows)
            assert s.wait(s.submit(i, x, y), 60.0)["status"] == 0
            want = to_dev(np.empty(mats[i].num_rows))
            L.LeSpMV(1.0, L.csr_from_host(mats[i]), to_dev(x), 0.0, want)
            assert np.array_equal(y, to_host(want))
        with pytest.raises(SSPMVError) as e:
            s.wait(s.submit(1, x, np.empty(mats[1].num_rows)), 60.0)
        assert e.value.status == 1
        st = s.stats()
        assert st["batched_requests"] == 1 and st["batched_tiles"] == 8
