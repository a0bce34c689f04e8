"""Two threads, each with a context of its own, launch the same norm kernels with row lengths in turn: the kernel's limit
of dynamic shared memory and the kept occupancies belong to both."""
import threading

import numpy as np
import pytest
import torch

import autograd_b200 as ag

pytestmark = pytest.mark.gpu

LENGTHS = [(1000, 768), (768, 1000), (1020, 512, 896)]   # (1 + 16) rows of floats: from 34 to 69 KB per CTA


def _backward(ctx, data, c):
    dy, x, gamma, part = data
    dx, dg, db = torch.zeros(200, c, device="cuda"), torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
    torch.cuda.synchronize()
    ctx.layernorm_backward(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), 0, dx.data_ptr(), dg.data_ptr(), db.data_ptr(),
                           part.data_ptr(), part.numel() * 4, 200, c, 1e-5)
    return dx, dg, db


def _work(lengths, rounds, out):
    ctx = ag.context.CudaContext(0)
    try:
        torch.manual_seed(sum(lengths))
        want, data = {}, {}
        for c in lengths:
            data[c] = (torch.randn(200, c, device="cuda"), torch.randn(200, c, device="cuda"), torch.randn(c, device="cuda"),
                       torch.empty(ctx.norm_partials_bytes(c) // 4, device="cuda"))
            want[c] = _backward(ctx, data[c], c)
        ctx.synchronize()
        for _ in range(rounds):
            for c in lengths:
                got = _backward(ctx, data[c], c)
                ctx.synchronize()
                for a, b in zip(got, want[c]):
                    if not torch.equal(a, b):
                        raise AssertionError(f"{c} columns: another result")
        out.append(None)
    except BaseException as e:  # reported by the test's own thread
        out.append(e)
    finally:
        ctx.close()


def test_row_lengths_in_turn_from_two_threads():
    out = []
    threads = [threading.Thread(target=_work, args=(lengths, 60, out)) for lengths in LENGTHS]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(out) == len(LENGTHS)
    for e in out:
        if e is not None:
            raise e
    assert np.all([e is None for e in out])
