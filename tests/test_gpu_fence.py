"""Ordering of the library's stream against the caller's (spmv_comm_fence) and
new values given as device memory: results on a side stream and from several
threads are those of a call that waits, and the host copy of the values
follows the device's."""
import threading

import numpy as np
import pytest
import torch

import oracle
from spmv_b200 import gen
from helpers import build

pytestmark = pytest.mark.gpu


def test_fence_on_side_streams_and_threads(cuda_device):
    W = gen.workload("c2", 48)
    comm, cm, rm, M, D = build(W, 3)
    rng = np.random.default_rng(0)
    base = [rng.standard_normal(cm.vec_len(q)) for q in range(3)]
    errors = []

    def worker(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for rep in range(20):
                    scale = float(1 + i + rep)
                    # Work queued ahead of the inputs, so a call that did not
                    # wait for this stream would read the old ones.
                    xs = [torch.zeros(len(b), dtype=torch.float64, device="cuda") for b in base]
                    torch.cuda._sleep(200000)
                    for x, b in zip(xs, base):
                        x.add_(torch.from_numpy(b).cuda() * scale)
                    ys = [2.0 * y for y in M.mult(xs)]
                    s.synchronize()
                    for q in range(3):
                        rp, ci, va = D.blocks[q]
                        ref = 2.0 * oracle.csr_mult(rp, ci, va, base[q] * scale)
                        assert np.array_equal(ys[q].cpu().numpy(), ref)
        except BaseException as e:  # noqa: BLE001 - reported by the test thread
            errors.append(e)

    M.mult([torch.from_numpy(b).cuda() for b in base])  # layouts are built once
    torch.cuda.synchronize()
    threads = [threading.Thread(target=worker, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_default_stream_calls_between_host_calls_and_the_handle(cuda_device):
    """Calls that run on the default stream itself, host-vector calls on the
    library's stream and work the caller puts on its handle, in turn: each
    sees what was before it."""
    W = gen.workload("c2", 40)
    comm, cm, rm, M, D = build(W, 4)
    rng = np.random.default_rng(1)
    xh = [rng.standard_normal(cm.vec_len(q)) for q in range(4)]
    ref = [oracle.csr_mult(*D.blocks[q], xh[q]) for q in range(4)]

    def same(ys):
        torch.cuda.synchronize()
        return all(np.array_equal(y.cpu().numpy() if torch.is_tensor(y) else y, r)
                   for y, r in zip(ys, ref))

    for handed_out in (False, True):
        for _ in range(5):
            xs = [torch.zeros(len(v), dtype=torch.float64, device="cuda") for v in xh]
            src = [torch.from_numpy(v).cuda() for v in xh]
            torch.cuda._sleep(1000000)
            for x, v in zip(xs, src):
                x.copy_(v)
            ys = M.mult(xs)                       # on the default stream, or fenced
            zs = [y + 0.0 for y in ys]
            assert same(M.mult(xh))               # host vectors: the library's stream
            assert same(zs)
            M.set_values([va * 2.0 for _, _, va in D.blocks])
            M.set_values([va for _, _, va in D.blocks])
            assert same(M.mult(xs))
        if not handed_out:
            ts = comm.torch_stream()
            assert ts.cuda_stream == comm.stream
    with torch.cuda.stream(ts):
        assert same(M.mult([torch.from_numpy(v).cuda() for v in xh]))
    comm.synchronize()


def test_device_values_reach_the_host_copy_and_the_transpose(cuda_device):
    W = gen.workload("c1", 40)
    comm, cm, rm, M, D = build(W, 2)
    new = [np.random.default_rng(q).standard_normal(len(D.blocks[q][2])) for q in range(2)]
    M.set_values([torch.from_numpy(v).cuda() for v in new])
    for q in range(2):
        np.testing.assert_array_equal(M.mat(q)[2], new[q])
    M.set_values([torch.from_numpy(2.0 * v).cuda() for v in new])
    xs = [np.random.default_rng(9 + q).standard_normal(n) for q, n in enumerate(M.nrows)]
    ys = M.transpmult(xs)
    for q in range(2):
        rp, ci, _ = D.blocks[q]
        ref = oracle.csr_transpmult(rp, ci, 2.0 * new[q], xs[q], cm.vec_len(q))
        assert np.max(np.abs(ys[q] - ref)) <= 1e-12 * np.max(np.abs(ref))
    M.set_values(new)  # host values after device values
    np.testing.assert_array_equal(M.mat(1)[2], new[1])
