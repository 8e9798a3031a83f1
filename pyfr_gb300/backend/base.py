"""The ``b200`` backend: a GB300-native implementation of the reference's
backend interface (``pyfr/backends/base/backend.py:32-226`` with the
concrete attributes of ``pyfr/backends/cuda/base.py:9-144``).

One process drives one GPU through the pyfrb200 C ABI.  Matrices are
allocated in named extents, kernels are obtained from the providers by
name (``backend.kernel('mul', ...)``, ``backend.kernel('tflux', ...)``),
and graphs are captured as CUDA graphs.  There is no CPU fallback: if the
library or the GPU is missing, construction raises.
"""

from collections import namedtuple
from contextlib import contextmanager
import ctypes as C
import gc
import itertools as it
import weakref
from weakref import WeakValueDictionary

import numpy as np

from pyfr_gb300.backend import types
from pyfr_gb300.backend.lib import get_lib, B200Error


# Releases of device resources (graph executables, allocations, operator
# handles) requested while a stream capture was open: the runtime would
# invalidate the capture, and the finaliser of any backend's objects may
# run then.  Process-wide, run when the outermost capture ends.
_CAPTURE_DEPTH = 0
_DEFERRED = []


def release(fn, *args):
    """Call ``fn(*args)`` now, or once no stream capture is open."""
    if _CAPTURE_DEPTH:
        _DEFERRED.append((fn, args))
    else:
        fn(*args)


def _free_allocs(lib, allocs):
    for p, _ in allocs:
        try:
            lib.free(p)
        except B200Error:
            pass
    allocs.clear()

# Constants up to this many elements keep a host copy after set-up (for
# reuse of identical constants and for the operator handles)
HOST_KEEP = 1 << 20

MemoryInfo = namedtuple('MemoryInfo', ['current', 'peak', 'free', 'total'])


class NotSuitableError(Exception):
    pass


def _recordmat(fn):
    def newfn(self, *args, **kwargs):
        m = fn(self, *args, **kwargs)
        if not hasattr(m, 'mid'):
            m.mid = next(self._mat_counter)
            self.mats[m.mid] = m
        return m
    newfn.__name__ = fn.__name__
    return newfn


class B200Backend:
    name = 'b200'
    blocks = False
    has_double = True

    def __init__(self, cfg):
        self.cfg = cfg

        prec = cfg.get('backend', 'precision', 'double')
        if prec not in {'single', 'double'}:
            raise ValueError('Backend precision must be either single or '
                             'double')
        self.fpdtype = np.dtype(prec).type
        self.fpdtype_eps = float(np.finfo(self.fpdtype).eps)
        self.fpdtype_max = float(np.finfo(self.fpdtype).max)

        match cfg.get('backend', 'memory-model', 'normal'):
            case 'normal':
                self.ixdtype = np.int32
            case 'large':
                self.ixdtype = np.int64
            case _:
                raise ValueError('Backend memory model must be either normal '
                                 'or large')

        self.autotune_ifac = cfg.getfloat('backend', 'autotune-ifac', 0.95)

        # Layout constants (as the reference CUDA backend)
        self.alignb = 128
        self.soasz = 32
        self.csubsz = self.soasz

        # Execution options of this backend
        self.use_cuda_graphs = cfg.getbool('backend-b200', 'cuda-graphs', True)
        self.fusion = cfg.getbool('backend-b200', 'fusion', True)
        self.precompute_metrics = cfg.getbool('backend-b200',
                                              'precompute-metrics', True)
        # Affine elements keep one set of metric terms per element
        self.per_element_metrics = cfg.getbool('backend-b200',
                                               'per-element-metrics', True)
        # Constant (rho_ref, p_ref) that Navier-Stokes kernels subtract from
        # their inputs; set by the mixed-precision integrator before the
        # kernels are built (None: inputs are the conserved variables)
        self.ref_state = None
        self.mul_precision = cfg.get('backend-b200', 'mul-precision', 'native')
        if self.mul_precision not in {'native', 'bf16x3', 'tf32'}:
            raise ValueError('mul-precision must be native, bf16x3 or tf32')

        # Tensor-core pipeline plans picked by timing (cached per device
        # and operator); off: the deepest plan that fits
        self.autotune = cfg.get('backend-b200', 'autotune', 'true') == 'true'

        # Split-BF16 products: 3 (Ahi Bhi + Ahi Blo + Alo Bhi) or 4 (plus
        # Alo Blo)
        # 3: Ahi*Bhi + Ahi*Blo + Alo*Bhi; 4: plus Alo*Blo; 5: the operator in
        # three BF16 terms, plus Ax3*Bhi (operators whose three-term image
        # does not fit shared memory fall back to four products)
        self.split_products = cfg.getint('backend-b200', 'split-products', 3)
        if self.split_products not in {3, 4, 5}:
            raise ValueError('split-products must be 3, 4 or 5')

        # Fused operator applies (mul_cat, mul_batched): the tensor-core
        # provider serves them, so by default they follow mul-precision
        fuse = cfg.get('backend-b200', 'fuse-operators', 'auto')
        if fuse not in {'auto', 'true', 'false'}:
            raise ValueError('fuse-operators must be auto, true or false')
        tensor = (self.mul_precision in {'bf16x3', 'tf32'} and
                  self.fpdtype == np.float32)
        if fuse == 'true' and not tensor:
            raise ValueError('fuse-operators needs single precision with '
                             'mul-precision = bf16x3 or tf32')
        self.fuse_operators = tensor and fuse != 'false'

        # The mixed-precision RK stage in the epilogue of the divergence
        # apply (with fused operator applies).  Off unless asked for: the
        # epilogue's FP64 read-modify-write is latency-bound (one thread per
        # column walks its rows), and at the 48^3 benchmark the step runs
        # 11% slower with it than with the separate stage kernel
        fstage = cfg.get('backend-b200', 'fuse-stage', 'auto')
        if fstage not in {'auto', 'true', 'false'}:
            raise ValueError('fuse-stage must be auto, true or false')
        self.fuse_stage = self.fuse_operators and fstage == 'true'

        self.mats = WeakValueDictionary()
        self._mat_counter = it.count()
        self._extents = {}
        self._allocs = []
        self._mem_cur = self._mem_peak = 0

        # Bring up the device
        self.lib = lib = get_lib()
        devid = cfg.get('backend-b200', 'device-id', '0')
        lib.init(int(devid))

        s = C.c_void_p()
        lib.stream_create(C.byref(s))
        self._stream = s.value

        # Device memory goes back when the backend is collected
        weakref.finalize(self, release, _free_allocs, lib, self._allocs)

        self.const_matrix_cls = types.ConstMatrix
        self.matrix_cls = types.Matrix
        self.matrix_slice_cls = types.MatrixSlice
        self.xchg_matrix_cls = types.XchgMatrix
        self.view_cls = types.View
        self.xchg_view_cls = types.XchgView
        self.graph_cls = types.Graph
        self.ordered_meta_kernel_cls = types.OrderedMetaKernel
        self.unordered_meta_kernel_cls = types.UnorderedMetaKernel

        # Element kernels of tensor-product elements (tensorele.py) where
        # they apply; 'general': the operator applies and pointwise kernels
        # one by one
        self.element_kernels = cfg.get('backend-b200', 'element-kernels',
                                       'auto')
        if self.element_kernels not in {'auto', 'general'}:
            raise ValueError('element-kernels must be auto or general')

        from pyfr_gb300.backend import (blasext, fused, mul, pointwise,
                                        tensorele)
        self._providers = [pointwise.PointwiseKernelProvider(self),
                           blasext.BlasExtKernels(self),
                           mul.TensorMulKernels(self),
                           mul.MulKernels(self),
                           tensorele.TensorElementKernels(self)]
        self.pointwise = self._providers[0]
        self.tensor_elements = self._providers[-1]
        self._fuser = fused.Fuser(self)
        self._status = None

    # ---- device status word (pipeline timeouts inside kernels) -------------

    @property
    def status_word(self):
        """Device address of an int that kernels set on a bounded-wait
        timeout; 0 means no error."""
        if self._status is None:
            p = C.c_void_p()
            self.lib.malloc(C.byref(p), 16)
            self._status = p.value
        return self._status

    def check_status(self):
        """Raise if any kernel recorded a timeout since the last check."""
        if self._status is None:
            return
        v = np.zeros(1, dtype=np.int32)
        self.lib.memcpy_dtoh(v.ctypes.data, self._status, 4, self._stream)
        self.lib.stream_sync(self._stream)
        if v[0]:
            self.lib.memset(self._status, 0, 4, self._stream)
            raise B200Error(f'kernel pipeline timeout (code {int(v[0])})')

    # ---- device plumbing --------------------------------------------------

    @property
    def stream(self):
        return self._stream

    @property
    def platform_id(self):
        name = C.create_string_buffer(256)
        self.lib.device_info(None, None, None, None, None, name, 256)
        return name.value.decode()

    def _malloc_impl(self, nbytes):
        p = C.c_void_p()
        self.lib.malloc(C.byref(p), nbytes)
        self._allocs.append((p.value, nbytes))
        self._mem_cur += nbytes
        self._mem_peak = max(self._mem_peak, self._mem_cur)
        return p.value

    def free_matrix(self, m):
        """Release a matrix that owns its allocation (one made without a
        named extent); using it afterwards is an error."""
        for i, (p, n) in enumerate(self._allocs):
            if p == m.basedata and m.offset == 0:
                self.lib.free(p)
                self._mem_cur -= n
                del self._allocs[i]
                m.basedata = None
                return
        raise ValueError('Matrix does not own an allocation')

    def memcpy_htod(self, dst, src, nbytes):
        src = np.ascontiguousarray(src)
        self.lib.memcpy_htod(dst, src.ctypes.data, nbytes, self._stream)
        self.lib.stream_sync(self._stream)

    def memcpy_dtoh(self, dst, src, nbytes):
        self.lib.memcpy_dtoh(dst.ctypes.data, src, nbytes, self._stream)
        self.lib.stream_sync(self._stream)

    def wait(self):
        self.lib.stream_sync(self._stream)
        self.check_status()

    def memory_info(self):
        f, t = C.c_size_t(), C.c_size_t()
        self.lib.device_info(None, None, None, C.byref(f), C.byref(t), None, 0)
        return MemoryInfo(self._mem_cur, self._mem_peak, f.value, t.value)

    def capture(self, launch, stream):
        """Record ``launch(stream)`` into a CUDA graph and return its
        executable.  While a capture is open no graph or memory may be
        released (the runtime invalidates the capture), so the cyclic
        garbage collector, whose finalisers release graphs, is paused and
        releases requested meanwhile are deferred until the capture ends."""
        global _CAPTURE_DEPTH
        gc_was_enabled = gc.isenabled()
        gc.disable()
        _CAPTURE_DEPTH += 1
        try:
            self.lib.graph_begin_capture(stream)
            try:
                launch(stream)
            except BaseException:
                g = C.c_void_p()
                try:
                    self.lib.graph_end_capture(stream, C.byref(g))
                except B200Error:
                    pass
                else:
                    _DEFERRED.append((self.lib.graph_destroy, (g.value,)))
                raise
            g = C.c_void_p()
            self.lib.graph_end_capture(stream, C.byref(g))
            return g.value
        finally:
            _CAPTURE_DEPTH -= 1
            if not _CAPTURE_DEPTH:
                while _DEFERRED:
                    fn, args = _DEFERRED.pop()
                    fn(*args)
            if gc_was_enabled:
                gc.enable()

    def launcher(self, nodes):
        """A function enqueueing ``nodes`` on a stream that is being
        captured: a list of kernels, one after the other, or ``types.Nodes``,
        each of which the graph then starts when those that it waits for
        have finished (the capture's own dependencies are set before each
        kernel: no other streams, no events)."""
        if not isinstance(nodes, types.Nodes):
            def launch(stream):
                for k in nodes:
                    k.run(stream)
            return launch

        last, after = self.lib.graph_capture_last, self.lib.graph_capture_after
        items = nodes.by_chains()
        # (a node that waits for the one before it alone follows it anyway)
        chained = [n > 0 and deps == [items[n - 1][1]]
                   for n, (_, _, deps) in enumerate(items)]
        used = {d for (_, _, deps), c in zip(items, chained) if not c
                for d in deps}
        ends = set(range(len(items))) - {d for *_, deps in items for d in deps}
        used |= ends
        buf, n = (C.c_void_p*8)(), C.c_int()

        def launch(stream):
            def captured():
                last(stream, buf, len(buf), C.byref(n))
                return buf[:n.value]

            def follow(handles):
                after(stream, (C.c_void_p*max(len(handles), 1))(*handles),
                      len(handles))

            before, got = captured(), {}
            for j, (k, i, deps) in enumerate(items):
                if j and not chained[j]:
                    follow(sorted({h for d in deps for h in got[d]})
                           if deps else before)
                k.run(stream)
                if i in used:
                    got[i] = captured()
            follow(sorted({h for i in ends for h in got[i]}))

        return launch

    def release_gexec(self, gexec):
        if gexec:
            release(self.lib.graph_destroy, gexec)

    # ---- allocation (pyfr/backends/base/backend.py:94-165) ----------------

    def _extent_alloc_bytes(self, nbytes):
        return nbytes - (nbytes % -self.alignb)

    def malloc(self, obj, extent):
        if extent is None:
            ext = types.Extent()
            ext.reserve(obj, self._extent_alloc_bytes(obj.nbytes))
            ext.commit(self._malloc_checked)
        else:
            ext = self._extents.setdefault(extent, types.Extent(extent))
            ext.reserve(obj, self._extent_alloc_bytes(obj.nbytes))

    def commit(self):
        for ext in self._extents.values():
            ext.commit(self._malloc_checked)
        self._extents.clear()

    def _malloc_checked(self, nbytes):
        if self.ixdtype == np.int32 and nbytes > 4*2**31 - 1:
            raise RuntimeError('Allocation too large for normal backend '
                               'memory-model')
        return self._malloc_impl(nbytes)

    @_recordmat
    def const_matrix(self, initval, dtype=None, tags=set()):
        dtype = dtype or self.fpdtype
        initval = np.asarray(initval)

        # Reuse an identical constant (pyfr/backends/base/backend.py:134-145);
        # only small constants (operators) are compared
        for m in list(self.mats.values()) if initval.size <= HOST_KEEP else []:
            if (isinstance(m, self.const_matrix_cls) and
                m.dtype == np.dtype(dtype) and m.ioshape == initval.shape and
                set(tags).issubset(m.tags) and
                getattr(m, '_host', None) is not None and
                np.array_equal(m._host, initval)):
                return m

        m = self.const_matrix_cls(self, dtype, initval, tags)
        # The host copy keeps the precision it was given: host-side
        # computations from constants (metric terms from vertices, operator
        # splits) must not inherit the device precision's rounding
        m._host = np.array(initval)
        return m

    def release_host_copies(self):
        """Drop the host copies of large constants (geometry, gather maps):
        they serve the set-up only; operators keep theirs."""
        for m in list(self.mats.values()):
            h = getattr(m, '_host', None)
            if isinstance(m, self.const_matrix_cls) and h is not None and \
                    h.size > HOST_KEEP:
                del m._host

    @_recordmat
    def matrix(self, ioshape, initval=None, extent=None, tags=set(),
               dtype=None):
        dtype = dtype or self.fpdtype
        return self.matrix_cls(self, dtype, ioshape, initval, extent, tags)

    @_recordmat
    def matrix_slice(self, mat, ra, rb, ca, cb):
        return self.matrix_slice_cls(self, mat, ra, rb, ca, cb)

    @_recordmat
    def xchg_matrix(self, ioshape, initval=None, extent=None, tags=set()):
        return self.xchg_matrix_cls(self, self.fpdtype, ioshape, initval,
                                    extent, tags)

    def xchg_matrix_for_view(self, view, tags=set()):
        return self.xchg_matrix((view.nvrow, view.nvcol*view.n), tags=tags)

    def view(self, matmap, rmap, cmap, rstridemap=1, vshape=(), tags=set()):
        return self.view_cls(self, matmap, rmap, cmap, rstridemap, vshape,
                             tags)

    def xchg_view(self, matmap, rmap, cmap, rstridemap=1, vshape=(),
                  tags=set()):
        return self.xchg_view_cls(self, matmap, rmap, cmap, rstridemap,
                                  vshape, tags)

    # ---- kernels (pyfr/backends/base/backend.py:177-226) ------------------

    @contextmanager
    def region(self, name):
        yield

    def kernel(self, name, *args, **kwargs):
        best = None
        for prov in self._providers:
            meth = getattr(prov, name, None)
            if meth is None:
                continue
            try:
                kern = meth(*args, **kwargs)
            except NotSuitableError:
                continue

            if best is None or kern.dt < self.autotune_ifac*best.dt:
                best = kern
                if np.isnan(best.dt):
                    return best

        if best is None:
            raise KeyError(f'Kernel {name!r} has no providers')
        return best

    def ordered_meta_kernel(self, kerns):
        return self.ordered_meta_kernel_cls(kerns)

    def unordered_meta_kernel(self, kerns, splits=None):
        return self.unordered_meta_kernel_cls(kerns, splits)

    def graph(self):
        return self.graph_cls(self)

    def fuse(self, klist, groups):
        return self._fuser.fuse(klist, groups) if self.fusion else klist

    def run_kernels(self, kernels, wait=False):
        for k in kernels:
            k.run(self._stream)
        if wait:
            self.wait()

    def run_graph(self, graph, wait=False):
        graph.run(self._stream)
        if wait:
            self.wait()
