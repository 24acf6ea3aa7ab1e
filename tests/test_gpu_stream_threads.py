"""Products of one communicator from several threads, on torch's default stream
(where the library works on it directly) and on a side stream: every result is
that of the thread's own inputs, and no thread waits for another for good."""
import threading

import numpy as np
import pytest
import torch

import oracle
from spmv_b200 import gen
from helpers import build

pytestmark = pytest.mark.gpu


def test_default_and_side_streams_at_once(cuda_device):
    W = gen.workload("c2", 40)
    comm, cm, rm, M, D = build(W, 3)
    rng = np.random.default_rng(0)
    base = [rng.standard_normal(cm.vec_len(q)) for q in range(3)]
    M.mult([torch.from_numpy(b).cuda() for b in base])  # layouts are built once
    refs = [oracle.csr_mult(*D.blocks[q], base[q]) for q in range(3)]
    torch.cuda.synchronize()
    errors, done = [], []

    def worker(i):
        try:
            stream = torch.cuda.Stream() if i == 2 else torch.cuda.default_stream()
            with torch.cuda.stream(stream):
                for rep in range(40):
                    scale = float(2 ** ((i + rep) % 5))
                    xs = [torch.from_numpy(b).cuda() * scale for b in base]
                    ys = M.mult(xs)
                    stream.synchronize()
                    for y, ref in zip(ys, refs):
                        assert np.array_equal(y.cpu().numpy(), scale * ref)
            done.append(i)
        except BaseException as e:  # noqa: BLE001 - reported by the test thread
            errors.append(e)

    threads = [threading.Thread(target=worker, args=(i,), daemon=True) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors[0]
    assert sorted(done) == [0, 1, 2]
