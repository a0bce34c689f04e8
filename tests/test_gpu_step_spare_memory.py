"""A step that does without the memory that only saves time: the gradients of one that has it, to rounding, with no error left
behind by the allocation that failed."""
import numpy as np
import pytest

import gpu_util as G
from autograd_b200 import _native as N
from autograd_b200.step import FusedLayerStep, StepConfig
from autograd_b200.storage import CudaAllocator
from conftest import assert_close

pytestmark = pytest.mark.gpu


class _Allocator(CudaAllocator):
    """Asks the device for more than it has wherever a buffer of one of these sizes is wanted."""
    refuse = ()

    def alloc(self, shape, dtype=np.float32):
        if shape in [(n,) for n in self.refuse]:
            shape = (1 << 50,)
        return super().alloc(shape, dtype)


@pytest.mark.parametrize("precision", [N.AG_CE_3XTF32, N.AG_CE_BF16X3])
@pytest.mark.parametrize("seq,vocab", [(40, 392), (1400, 4104)])     # a short head and one on operand pairs
def test_step_without_spare_memory(seq, vocab, precision):
    ctx, _, be = G.env()
    cfg = StepConfig(n_layer=2, n_embd=512, n_head=4, head_dim=128, seq_len=seq, vocab=vocab, batch=3, ce_precision=precision)
    rng = np.random.default_rng(seq)
    ids, targets = rng.integers(0, vocab, (2, 3 * seq)).astype(np.int32)
    got = []
    for spare in (True, False):
        alloc = _Allocator(ctx)
        desc = ctx.flce_desc(3 * seq, 512, vocab, precision=precision)
        if not spare:
            alloc.refuse = (ctx.flce_logits_bytes(desc), 5 * ctx.norm_partials_bytes(512))
        st = FusedLayerStep(ctx, alloc, be, cfg, seed=3)
        assert (st._batch, st.logits is None) == ((5, False) if spare else (1, True))
        ctx.copy_from_host(st.ids, ids)
        ctx.copy_from_host(st.targets, targets)
        for _ in range(3):        # launched, recorded, replayed
            st.step()
        got.append([ctx.copy_to_host(a, (n,), np.float32).copy() for a, n in
                    ((st.small_bucket, st.n_small + 1), (st.dtable, st.V * st.C), (st.dh, st.N * st.C))])
        G.check_clean_status()
        st.close()
    free, total = ctx.memory()
    assert 0 < free < total == ctx.total_bytes
    for a, b in zip(*got):        # both are within 1e-4 of the exact gradient (what the tests of the head ask of each)
        assert np.isfinite(a).all() and a.any()
        assert_close(a.astype(np.float64), b.astype(np.float64), 2e-4, "gradients")
