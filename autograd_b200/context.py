"""`CudaContext`: the Python face of one `ag_ctx` (device + stream), the counterpart of the
reference's `metal_ext.MetalContext` (metal_ext.mm:770-796).  Methods take raw device
addresses (ints) and sizes; they map one to one onto the C ABI.
"""
from __future__ import annotations

import ctypes as C

import numpy as np

from . import _native as N
from ._native import calls, lib


def _p(addr):
    """int / None -> c_void_p"""
    return C.c_void_p(int(addr)) if addr else C.c_void_p(0)


class CudaContext:
    def __init__(self, device: int = 0, stream: int | None = None):
        h = C.c_void_p()
        rc = lib.ag_ctx_create(int(device), _p(stream), C.byref(h))
        if rc != N.AG_OK:
            raise N.AgError(rc, (lib.ag_last_error(None) or b"").decode())
        self.eager = False  # GEMM timing is on: launches have to be made one by one
        self._h = h
        self._hi = h.value  # the same handle as the integer that `calls` takes
        self.device = int(device)
        sm, l2, tot, maj, mnr = C.c_int(), C.c_int64(), C.c_int64(), C.c_int(), C.c_int()
        self._check(lib.ag_device_info(h, C.byref(sm), C.byref(l2), C.byref(tot), C.byref(maj), C.byref(mnr)))
        self.sm_count, self.l2_bytes, self.total_bytes = sm.value, l2.value, tot.value
        self.compute_capability = (maj.value, mnr.value)

    # ------------------------------------------------------------------ plumbing
    def _check(self, rc):
        if rc != N.AG_OK:
            raise N.AgError(rc, (lib.ag_last_error(self._h) or b"").decode())

    def close(self):
        if getattr(self, "_h", None):
            lib.ag_ctx_destroy(self._h)
            self._h = None
            self._hi = 0

    def __del__(self):  # best effort
        try:
            self.close()
        except Exception:
            pass

    def set_stream(self, stream):
        self._check(lib.ag_set_stream(self._h, _p(stream)))

    def memory(self):
        """(free, total) bytes of the device."""
        free, total = C.c_int64(), C.c_int64()
        self._check(lib.ag_memory_info(self._h, C.byref(free), C.byref(total)))
        return free.value, total.value

    def alloc(self, nbytes: int) -> int:
        out = C.c_void_p()
        self._check(lib.ag_alloc(self._h, int(nbytes), C.byref(out)))
        return int(out.value or 0)

    def free(self, addr: int):
        self._check(lib.ag_free(self._h, _p(addr)))

    def copy_from_host(self, dst_addr: int, host: np.ndarray):
        host = np.ascontiguousarray(host)
        calls.ag_copy_h2d(self._hi, dst_addr, host.ctypes.data, host.nbytes)

    def copy_to_host(self, src_addr: int, shape, dtype) -> np.ndarray:
        out = np.empty(shape, dtype=dtype)
        self._check(lib.ag_copy_d2h(self._h, out.ctypes.data_as(C.c_void_p), _p(src_addr), out.nbytes))
        return out

    def copy_h2d_raw(self, dst_addr: int, host_addr: int, nbytes: int):
        calls.ag_copy_h2d(self._hi, dst_addr, host_addr, nbytes)

    def copy_d2h_raw(self, host_addr: int, src_addr: int, nbytes: int):
        self._check(lib.ag_copy_d2h(self._h, _p(host_addr), _p(src_addr), int(nbytes)))

    def synchronize(self):
        self._check(lib.ag_synchronize(self._h))

    def status(self) -> int:
        f = C.c_int()
        self._check(lib.ag_status(self._h, C.byref(f)))
        return f.value

    def check_status(self):
        f = self.status()
        if f:
            names = [n for n, b in (("BAD_INDEX", 1), ("WAIT_EXPIRED", 2), ("STAGE_FALLBACK", 4)) if f & b]
            raise N.AgError(N.AG_ERR_DEVICE, "device status word: " + "|".join(names))

    @property
    def launch_count(self) -> int:
        return int(lib.ag_launch_count(self._h))

    def begin_pass_profiled(self):
        self._check(lib.ag_pass_begin_profiled(self._h))

    def end_pass_profiled(self) -> float:
        ms = C.c_float()
        self._check(lib.ag_pass_end_profiled(self._h, C.byref(ms)))
        return ms.value

    def event_record(self, index: int):
        calls.ag_event_record(self._hi, index)

    def event_elapsed_ms(self, start_index: int, end_index: int) -> float:
        ms = C.c_float()
        self._check(lib.ag_event_elapsed(self._h, int(start_index), int(end_index), C.byref(ms)))
        return ms.value

    # A recorded sequence of launches (see the header)
    def record(self, fn) -> int:
        """Handle of the launches that fn(recorder) makes on the recorder, a context of this device.  AgError with
        AG_ERR_CAPTURING, and nothing done, while the context's stream is being captured."""
        h, out = C.c_void_p(), C.c_void_p()
        self._check(lib.ag_graph_begin(self._h, C.byref(h)))
        recorder = CudaContext.__new__(CudaContext)
        recorder.__dict__.update(self.__dict__, _h=h, _hi=h.value)
        try:
            fn(recorder)
        except BaseException:
            if lib.ag_graph_end(self._h, h, C.byref(out)) == N.AG_OK:  # a part of the launches: of no use
                lib.ag_graph_destroy(self._h, out)
            raise
        finally:
            recorder._h = None
        self._check(lib.ag_graph_end(self._h, h, C.byref(out)))
        return int(out.value)

    def replay(self, graph: int):
        calls.ag_graph_launch(self._hi, graph)

    def drop_recording(self, graph: int):
        self._check(lib.ag_graph_destroy(self._h, _p(graph)))

    def tc_timing(self, enable: bool, first_event_index: int = 0):
        """Bracket every tensor-core GEMM launch of the CE head with pool events (see the header)."""
        self.eager = bool(enable)
        self._check(lib.ag_tc_timing(self._h, 1 if enable else 0, int(first_event_index)))

    def tc_timing_count(self) -> int:
        return int(lib.ag_tc_timing_count(self._h))

    def alloc_host(self, nbytes: int) -> int:
        out = C.c_void_p()
        self._check(lib.ag_alloc_host(self._h, int(nbytes), C.byref(out)))
        return int(out.value or 0)

    def free_host(self, addr: int):
        self._check(lib.ag_free_host(self._h, _p(addr)))

    # ------------------------------------------------------------------ kernels
    def fill_f32(self, dst, value, n):
        calls.ag_fill_f32(self._hi, dst, value, n)

    def fill_pattern(self, dst, pattern, itemsize, n):
        calls.ag_fill_pattern(self._hi, dst, pattern & 0xFFFFFFFF, itemsize, n)

    def add_forward(self, x, y, out, n):
        calls.ag_add_forward(self._hi, x, y, out, n)

    def add_backward(self, g, xgrad, ygrad, n):
        calls.ag_add_backward(self._hi, g, xgrad, ygrad, n)

    def add_layernorm_forward(self, x, r, gamma, beta, h, y, mean, rstd, N_, C_, eps):
        calls.ag_add_layernorm_forward(self._hi, x, r, gamma, beta, h, y, mean, rstd, N_, C_, eps)

    def zero_ranges(self, a, na, b, nb, c, nc):
        calls.ag_zero_ranges(self._hi, a, na, b, nb, c, nc)

    def layernorm_backward_rows(self, dy, x, gamma, dres, dx, partials, partials_bytes, rows, N_, C_, eps):
        """The number of partial rows goes to the int32 at host address `rows`."""
        calls.ag_layernorm_backward_rows(self._hi, dy, x, gamma, dres, dx, partials, partials_bytes, rows, N_, C_, eps)

    def norm_partials_add(self, partials, stride, rows, n, C_, out):
        calls.ag_norm_partials_add(self._hi, partials, stride, rows, n, C_, out)

    def norm_partials_bytes(self, C_):
        return calls.ag_norm_partials_bytes(self._hi, C_)

    def layernorm_backward(self, dy, x, gamma, dres, dx, dgamma, dbeta, partials, partials_bytes, N_, C_, eps):
        calls.ag_layernorm_backward(self._hi, dy, x, gamma, dres, dx, dgamma, dbeta, partials, partials_bytes, N_, C_,
                                    eps)

    def layernorm_backward_noalloc(self, dy, x, gamma, dres, dx, dgamma, dbeta, N_, C_, eps):
        """LayerNorm backward whose partial-sum workspace lives inside the library: for callers
        that cannot hand over (or allocate) scratch memory.  C_ <= 4096."""
        calls.ag_layernorm_backward_noalloc(self._hi, dy, x, gamma, dres, dx, dgamma, dbeta, N_, C_, eps)

    def debug_expire_staging(self):
        """Test hook: the next norm kernel gives up its staging wait at once (see the header)."""
        self._check(lib.ag_debug_expire_staging(self._h))

    def rmsnorm_forward(self, x, gamma, y, inv_rms, N_, C_, eps, dtype=N.AG_F32):
        calls.ag_rmsnorm_forward(self._hi, x, gamma, y, inv_rms, N_, C_, eps, dtype)

    def rmsnorm_backward(self, dz, x, gamma, dres, dx, dgamma, partials, partials_bytes, N_, C_, eps, dtype=N.AG_F32):
        calls.ag_rmsnorm_backward(self._hi, dz, x, gamma, dres, dx, dgamma, partials, partials_bytes, N_, C_, eps,
                                  dtype)

    def gelu_forward(self, x, y, n):
        calls.ag_gelu_forward(self._hi, x, y, n)

    def gelu_backward(self, x, dy, dres, dx, n):
        calls.ag_gelu_backward(self._hi, x, dy, dres, dx, n)

    def swiglu_forward(self, gu, hidden, N_, I_, dtype=N.AG_F32):
        calls.ag_swiglu_forward(self._hi, gu, hidden, N_, I_, dtype)

    def swiglu_backward(self, gu, dhidden, N_, I_, dtype=N.AG_F32):
        calls.ag_swiglu_backward(self._hi, gu, dhidden, N_, I_, dtype)

    def rope_qk(self, q, k, cos, sin, B, T, H, HKV, D, q_token_stride=None, k_token_stride=None, sin_sign=1,
                dtype=N.AG_F32):
        qs = H * D if q_token_stride is None else q_token_stride
        ks = HKV * D if k_token_stride is None else k_token_stride
        calls.ag_rope_qk(self._hi, q, k, cos, sin, B, T, H, HKV, D, qs, ks, sin_sign, dtype)

    def gather_forward(self, ids, table, out, n_ids, C_, V_):
        calls.ag_gather_forward(self._hi, ids, table, out, n_ids, C_, V_)

    @staticmethod
    def scatter_add_scratch_bytes(n_ids, C_, V_):
        return calls.ag_scatter_add_scratch_bytes(n_ids, C_, V_)

    def gather_backward(self, ids, dout, dtable, scratch, scratch_bytes, n_ids, C_, V_):
        calls.ag_gather_backward(self._hi, ids, dout, dtable, scratch, scratch_bytes, n_ids, C_, V_)

    def gather_backward_bf16(self, ids, dout, dtable_bits, scratch, scratch_bytes, n_ids, C_, V_):
        """Table gradient kept as bf16 bit patterns: row = bf16(float(row) + fp32 sum of its dout rows)."""
        calls.ag_gather_backward_bf16(self._hi, ids, dout, dtable_bits, scratch, scratch_bytes, n_ids, C_, V_)

    def f32_to_bf16(self, src, dst_bits, n, accumulate=False):
        calls.ag_f32_to_bf16(self._hi, src, dst_bits, n, 1 if accumulate else 0)

    def bf16_to_f32(self, src_bits, dst, n):
        calls.ag_bf16_to_f32(self._hi, src_bits, dst, n)

    @staticmethod
    def flce_desc(N_, C_, V_, vocab_chunk=4096, precision=N.AG_CE_3XTF32, reduction=N.AG_CE_MEAN_ALL_ROWS,
                  ignore_mode=N.AG_CE_IGNORE_MASKED):
        return N.FlceDesc(int(N_), int(C_), int(V_), int(vocab_chunk), int(precision), int(reduction),
                          int(ignore_mode))

    @staticmethod
    def flce_scratch_bytes(desc):
        return calls.ag_flce_scratch_bytes(desc)

    def flce_forward(self, desc, X, W, targets, row_scale, loss, lse, scratch, scratch_bytes):
        calls.ag_flce_forward(self._hi, desc, X, W, targets, row_scale, loss, lse, scratch, scratch_bytes)

    def flce_backward(self, desc, X, W, targets, row_scale, dloss, lse, dX, dW, scratch, scratch_bytes):
        calls.ag_flce_backward(self._hi, desc, X, W, targets, row_scale, dloss, lse, dX, dW, scratch, scratch_bytes)

    @staticmethod
    def flce_logits_bytes(desc):
        return calls.ag_flce_logits_bytes(desc)

    def flce_forward_keep(self, desc, X, W, targets, row_scale, loss, lse, logits, logits_bytes, scratch, scratch_bytes):
        calls.ag_flce_forward_keep(self._hi, desc, X, W, targets, row_scale, loss, lse, logits, logits_bytes, scratch,
                                   scratch_bytes)

    def flce_backward_kept(self, desc, X, W, targets, row_scale, dloss, lse, logits, logits_bytes, dX, dW, scratch,
                           scratch_bytes):
        calls.ag_flce_backward_kept(self._hi, desc, X, W, targets, row_scale, dloss, lse, logits, logits_bytes, dX, dW,
                                    scratch, scratch_bytes)

    @staticmethod
    def linear_add_scratch_bytes(N_, K_, C_, precision=N.AG_CE_3XTF32):
        return calls.ag_linear_add_scratch_bytes(N_, K_, C_, precision)

    def linear_add_forward(self, x, act, w, b, out, N_, K_, C_, precision, scratch, scratch_bytes):
        calls.ag_linear_add_forward(self._hi, x, act, w, b, out, N_, K_, C_, precision, scratch, scratch_bytes)

    def linear_add_backward(self, dout, act, w, dx, dact, dw, db, N_, K_, C_, precision, scratch, scratch_bytes):
        calls.ag_linear_add_backward(self._hi, dout, act, w, dx, dact, dw, db, N_, K_, C_, precision, scratch,
                                     scratch_bytes)

    def adamw_step(self, p, g, m, v, n, lr, lr_t, b1, b2, eps, weight_decay, grad_scale=1.0, grad_bf16=False):
        fn = calls.ag_adamw_step_bf16grad if grad_bf16 else calls.ag_adamw_step
        fn(self._hi, p, g, m, v, n, lr, lr_t, b1, b2, eps, weight_decay, grad_scale)
