"""The tensor-core operator kernel where its epilogue sets take whole tiles
(an odd number of 32-row groups) and where they share a tile's groups: against
the FP64 product, for one, two and several tiles a CTA.

Bound: the data is held in 16 significant bits (a relative residual of at most
2^-17), the operator in 16 or 24, and three products leave out one of 2^-18:
below 2^-15 in all, with the FP32 sums' 2^-23 a term.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lib():
    from pyfr_gb300.backend import B200Backend
    from pyfr_gb300.inifile import Inifile

    return B200Backend(Inifile()).lib


def _handle(lib, a, nterms):
    h, smem = C.c_void_p(), C.c_size_t()
    m, k = a.shape
    lib.mul_tc_create_terms(a.ctypes.data_as(C.POINTER(C.c_double)), k, None,
                            0, m, 0, nterms, 0, 0, C.byref(h), C.byref(smem))
    return h


@pytest.mark.parametrize('rk', [False, True])
@pytest.mark.parametrize('products', [3, 5])
@pytest.mark.parametrize('ncol', [4, 128, 19460, 152*128*3 + 132, 100004])
@pytest.mark.parametrize('m,k', [(1, 16), (20, 40), (32, 32), (33, 20),
                                 (65, 27), (96, 64), (128, 33)])
def test_epilogue_sets(m, k, ncol, products, rk):
    import torch

    from pyfr_gb300.backend.lib import MulArgs

    lib = _lib()
    rng = np.random.default_rng(m + ncol)
    a = rng.standard_normal((m, k))
    b = torch.from_numpy(rng.random((k, ncol)) - 0.25).float().cuda()
    c = torch.from_numpy(rng.random((m, ncol))).float().cuda()
    acc = c.double()
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    ad = torch.from_numpy(a).cuda()
    ref, mag = ad @ b.double(), ad.abs() @ b.double().abs()
    rb = (2.0**-15 + k*2.0**-23)*mag
    h = _handle(lib, a, 3 if products == 5 else 2)

    for beta in ([0.0] if rk else [0.0, 1.0]):
        out = c.clone()
        p = MulArgs(b1=b.data_ptr(), ldb1=ncol, c=out.data_ptr(), ldc=ncol,
                    ncol=ncol, nbatch=1, alpha=1.0, beta=beta,
                    products=products, err=err.data_ptr())
        if rk:
            p.rk_stage, p.rk_dt, p.rk_a, p.rk_b = 1, 0.5, 0.25, 2.0
            p.rk_acc, p.rk_u = acc.data_ptr(), out.data_ptr()
        torch.cuda.synchronize()
        lib.mul_bf16x3_apply(h, C.addressof(p), None)
        torch.cuda.synchronize()
        assert err.item() == 0
        if rk:
            # acc + dt b R and fl32(acc) + dt a R
            assert bool(((acc - (c.double() + ref)).abs() <= rb).all())
            want, tol = c.double() + 0.125*ref, 0.125*rb
        else:
            want, tol = ref + beta*c.double(), rb
        tol = tol + 2.0**-22*(want.abs() + mag)
        assert bool(((out.double() - want).abs() <= tol).all())
    lib.mul_bf16x3_destroy(h)


@pytest.mark.parametrize('nbatch', [1, 3])
@pytest.mark.parametrize('ncol', [4, 8640, 19460, 50000])
@pytest.mark.parametrize('rows', [(192, 183), (33, 40, 64), (96, 20, 64, 64),
                                  (20, 20, 20, 20, 20), (64, 65)])
def test_row_ranges_side_by_side(rows, ncol, nbatch):
    """Row ranges, each of two pieces along K (the first stored, the second
    added), in one call against the same applies one by one: the same bits,
    whether or not the ranges' kernels are alike."""
    import torch

    from pyfr_gb300.backend.lib import MulArgs

    lib = _lib()
    rng = np.random.default_rng(sum(rows) + ncol)
    m, ks = sum(rows), (40, 27)
    b = torch.from_numpy(rng.random((nbatch, sum(ks), ncol)) - 0.25)
    b = b.float().cuda()
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    out = [torch.full((nbatch, m, ncol), 7.0, device='cuda') for _ in '12']
    hs, calls = [], [[], []]
    for k0, k, beta in ((0, ks[0], 0.0), (ks[0], ks[1], 1.0)):
        r0 = 0
        for r in rows:
            h = _handle(lib, rng.standard_normal((r, k)), 2)
            hs.append(h)
            for o, cl in zip(out, calls):
                cl.append(MulArgs(
                    b1=b.data_ptr() + 4*k0*ncol, ldb1=ncol,
                    c=o.data_ptr() + 4*r0*ncol, ldc=ncol, ncol=ncol,
                    nbatch=nbatch, bstride1=sum(ks)*ncol, cstride=m*ncol,
                    alpha=0.5, beta=beta, products=4, err=err.data_ptr()))
            r0 += r
    n = len(hs)
    torch.cuda.synchronize()
    for h, a in zip(hs, calls[0]):
        lib.mul_bf16x3_apply(h, C.addressof(a), None)
    lib.mul_bf16x3_apply_pieces((C.c_void_p*n)(*(h.value for h in hs)),
                                (C.c_void_p*n)(*map(C.addressof, calls[1])),
                                n, None)
    torch.cuda.synchronize()
    assert err.item() == 0
    assert bool((out[0] == out[1]).all()) and bool((out[0] != 7.0).all())
    for h in hs:
        lib.mul_bf16x3_destroy(h)


@pytest.mark.parametrize('case', ['next slice', 'chained', 'in place', 'empty'])
def test_pieces_that_share_memory(case):
    """Pieces of which one writes what another reads or writes, in another
    slice or as its input, and a list with an empty piece, in one call against
    the same applies one by one: the same bits."""
    import torch

    from pyfr_gb300.backend.lib import MulArgs

    lib = _lib()
    rng = np.random.default_rng(8)
    m, k, ncol, nbatch = 32, 32, 8640, 2
    hs = [_handle(lib, rng.standard_normal((m, k)), 2) for _ in range(3)]
    b0 = torch.from_numpy(rng.random((nbatch + 2, k, ncol)) - 0.25).float()
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    sz, got = m*ncol, []
    for together in (False, True):
        b = b0.cuda()
        out = torch.zeros((nbatch + 2, m, ncol), device='cuda')

        def args(src, dst, beta=0.0, n=nbatch):
            return MulArgs(b1=src.data_ptr(), ldb1=ncol, c=dst.data_ptr(),
                           ldc=ncol, ncol=ncol, nbatch=n, bstride1=sz,
                           cstride=sz, alpha=0.5, beta=beta, products=3,
                           err=err.data_ptr())
        if case == 'next slice':
            # the second adds where the first's second slice is
            al = [args(b, out), args(b, out[1:], 1.0), args(b, out, 1.0)]
        elif case == 'chained':
            al = [args(b, out), args(out, out[nbatch:], 0.0),
                  args(b, out, 1.0)]
        elif case == 'in place':
            # the second writes what the first reads
            al = [args(b, out), args(out, b), args(b, out[nbatch:])]
        else:
            al = [args(b, out), args(b, out, n=0), args(b, out[nbatch:])]
        torch.cuda.synchronize()
        if together:
            n = len(al)
            lib.mul_bf16x3_apply_pieces(
                (C.c_void_p*n)(*(h.value for h in hs)),
                (C.c_void_p*n)(*map(C.addressof, al)), n, None)
        else:
            for h, a in zip(hs, al):
                lib.mul_bf16x3_apply(h, C.addressof(a), None)
        torch.cuda.synchronize()
        assert err.item() == 0
        got.append((out, b))
    assert all(bool((x == y).all()) for x, y in zip(*got))
    assert bool((got[0][0][:nbatch] != 0).any(-1).all())
    for h in hs:
        lib.mul_bf16x3_destroy(h)
