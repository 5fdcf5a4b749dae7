"""The chi**2 head at the edges of its row groups, point trips and kept curves.

Coefficients, components and mean are multiples of small powers of two, so the
FP32 curves are exact (every partial sum is a multiple of 2^-13 below 2); what
remains are double sums of npts terms: npts 2^-53 of the summed magnitudes, and
the scale's error enters chi**2 once more, twice: 4 npts 2^-53 bounds both.
"""
import ctypes as C
import os
import subprocess
import sys

import pytest

from lcurve_re_b200 import abi

pytestmark = pytest.mark.gpu


# 4096 points fit the kept curves; 2 rows a CTA, 512 points a trip
@pytest.mark.parametrize("rows,npts,nc", [(1, 1, 1), (2, 255, 64), (3, 512, 64), (5, 513, 100),
                                          (4, 4096, 16), (3, 4097, 16), (2, 9000, 7)])
@pytest.mark.parametrize("anchored", [False, True])
def test_chi2_of_exact_curves(rows, npts, nc, anchored):
    import torch
    from lcurve_re_b200.engine import load_library
    lib = load_library()
    g = torch.Generator(device="cuda").manual_seed(npts)

    def ints(lo, hi, *shape):
        return torch.randint(lo, hi + 1, shape, generator=g, device="cuda").float()
    coef, coef_x = ints(-4, 4, rows, nc) / 8, ints(-4, 4, rows, nc) / 8
    basis = ints(-8, 8, nc, npts) / 1024
    mean = 1 + ints(0, 800, npts) / 8192
    anchor = 1 + 0.1 * torch.rand(rows, npts, generator=g, device="cuda", dtype=torch.float64)
    flux = 1 + 0.1 * torch.rand(npts, generator=g, device="cuda", dtype=torch.float64)
    ferr = 0.1 + 0.1 * torch.rand(npts, generator=g, device="cuda", dtype=torch.float64)
    wgt = torch.rand(npts, generator=g, device="cuda", dtype=torch.float64)
    wgt[npts // 3] = 0.0 if npts > 1 else 1.0
    ferr[npts // 3] = 0.0 if npts > 1 else 0.1
    chi = torch.full((rows,), 7.0, dtype=torch.float64, device="cuda")
    sc = torch.full((rows,), 7.0, dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None
    st = lib.lcg_mlp_pca_chisq(C.c_void_p(torch.cuda.current_stream().cuda_stream), p(coef), rows,
                               nc, p(basis), p(mean), npts, p(flux), p(ferr), p(wgt),
                               p(coef_x) if anchored else None, p(anchor) if anchored else None,
                               p(chi), p(sc))
    torch.cuda.synchronize()
    assert st == abi.OK
    f = mean.double() + coef.double() @ basis.double()
    if anchored:
        f = anchor * (f / (mean.double() + coef_x.double() @ basis.double()))
    on = wgt > 0
    f, y, e, w = f[:, on], flux[on], ferr[on], wgt[on]
    s = (w / e ** 2 * y * f).sum(1) / (w / e ** 2 * f * f).sum(1)
    tol = 4 * (npts + 8) * 2.0 ** -53
    assert ((sc - s).abs() <= tol * s.abs()).all()
    want = (w * ((y - s[:, None] * f) / e) ** 2).sum(1)
    mag = (w * ((y.abs() + (s[:, None] * f).abs()) / e) ** 2).sum(1)
    assert ((chi - want).abs() <= tol * mag).all()


# curves and coefficients that fill the 48 KB a CTA has without asking, or all but the
# kernel's own static arrays; in a process of its own, since a kernel that was given
# more once keeps it
def test_chi2_at_the_default_shared_memory():
    sizes = [(2944, True), (3000, True), (3007, True), (3008, True), (3032, False), (3040, False)]
    code = "import test_gpu_pca_chisq as t\n" + "".join(
        "t.test_chi2_of_exact_curves(3, %d, 64, %s)\n" % s for s in sizes)
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                         env=env)
    assert out.returncode == 0, out.stderr[-2000:]
