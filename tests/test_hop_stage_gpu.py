"""The SIMT hop's epilogue vectors in shared memory: both staged (FP64 N = 2, FP32 N = 2, 3, 16-bit all
N but 4), x alone (FP64 N = 3, 4, FP32 N = 4..8 and 16-bit N = 4; none of the residual form) and none
(FP64 N >= 5), with m = 1, odd m whose block is not a multiple of 32 threads, m = 64 and half
volumes that leave the last blocks without sites; outputs and per-RHS sums against the oracle hop.

Tolerances: FP64 1e-13 of the output; FP32 sums at most 16 N + 2 terms per entry, 1e-6; 16-bit
storage computes in FP32 and rounds the output once, half a unit of its last place: 2^-11 and 2^-8
of each entry.  The per-RHS sums are those of the stored outputs: FP32 terms per thread, 1e-5, and
FP64 terms, 1e-12."""
import ctypes

import numpy as np
import pytest

import qcu_mrhs_b200 as q
from qcu_mrhs_b200 import fields as F
from tests.helpers import empty_dev, from_dev, rel_err, sync, to_dev

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [q.DOUBLE, q.SINGLE, q.HALF, q.BF16])
@pytest.mark.parametrize("L,nc,m", [((6, 2, 2, 2), 2, 7), ((2, 2, 2, 2), 3, 1), ((6, 4, 2, 6), 3, 13), ((4, 2, 2, 2), 3, 64),
                                   ((4, 4, 2, 2), 4, 5), ((4, 2, 4, 2), 5, 3), ((2, 4, 2, 2), 6, 9), ((4, 2, 2, 2), 8, 4)])
def test_staged_epilogues(oracle_lib, L, nc, m, prec):
    a = 0.0121
    rnd = lambda v: from_dev(to_dev(v, prec))   # the values as they are stored
    gauge = F.gauge_field(L, nc, 50 + nc)
    inp, x, r0 = (rnd(F.to_mrhs(F.gaussian_fermions(L, nc, m, 51 + i, parities=1)[:, 0])) for i in range(3))
    hop = oracle_lib.hop(inp, rnd(gauge), L, 1, False, -1.0)
    grid = q.QcuGrid((ctypes.c_int * 4)(1, 1, 1, 1))
    param = q.QcuParam((ctypes.c_int * 4)(*L))
    lib = q.lib()
    lib.initGridSize(ctypes.byref(grid), ctypes.byref(param), nc, m, q.DOUBLE, q.DOUBLE)
    q.check()
    dg = to_dev(gauge)
    lib.loadQcuGauge(dg.data_ptr(), q.DOUBLE)
    lib.getDslash(0, 0.5)
    o = q.default_options()
    o.t_boundary = -1.0
    q.check(lib.qcuSetSolverOptions(ctypes.byref(o)))
    q.check(lib.qcuSetHopKernel(q.HOP_SIMT))
    tol = {q.DOUBLE: 1e-13, q.SINGLE: 1e-6, q.HALF: 2.0 ** -11, q.BF16: 2.0 ** -8}[prec]
    stol = 1e-12 if prec == q.DOUBLE else 1e-5
    try:
        d_in, d_x, d_r0 = to_dev(inp, prec), to_dev(x, prec), to_dev(r0, prec)
        for form in (q.HOP_FORM_XPAY, q.HOP_FORM_SCHUR_R0, q.HOP_FORM_SCHUR_TS, q.HOP_FORM_SCHUR, q.HOP_FORM_RESID):
            d_out = empty_dev(inp.shape, prec)
            red = torch.zeros((2 * m, 2), dtype=torch.float64, device="cuda")
            q.check(lib.qcuDslashMrhsContextForm(d_out.data_ptr(), d_in.data_ptr(), d_x.data_ptr(), d_r0.data_ptr(),
                                                 a, form, 1, prec, red.data_ptr(), None))
            sync()
            got = from_dev(d_out)
            want = {q.HOP_FORM_XPAY: x + a * hop, q.HOP_FORM_RESID: r0 - (x - a * hop)}.get(form, x - a * hop)
            assert rel_err(got, want) <= tol
            sums = red.cpu().numpy()
            sums = sums[:, 0] + 1j * sums[:, 1]
            flat = lambda v: v.reshape(-1, m)
            norms = np.sqrt(np.sum(np.abs(flat(got)) ** 2, axis=0))
            if form == q.HOP_FORM_SCHUR_R0:
                ref = np.sum(np.conj(flat(r0)) * flat(got), axis=0)
                assert np.all(np.abs(sums[:m] - ref) <= stol * norms * np.linalg.norm(flat(r0), axis=0))
            elif form == q.HOP_FORM_SCHUR_TS:
                ref = np.sum(np.conj(flat(got)) * flat(x), axis=0)
                assert np.all(np.abs(sums[:m] - ref) <= stol * norms * np.linalg.norm(flat(x), axis=0))
                assert np.allclose(sums[m:2 * m].real, norms ** 2, rtol=stol)
            elif form == q.HOP_FORM_RESID:
                assert np.allclose(sums[:m].real, norms ** 2, rtol=stol)
    finally:
        lib.qcuSetHopKernel(q.HOP_AUTO)
        lib.finalizeQcu()
