"""The y and z passes whose lines stay inside a warp, against the oracle: every
line length they take, with few z lines (one-warp CTAs) and with many (several
warps per CTA), through the plain transforms and the three solvers' steps."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from tests.conftest import rel_l2
from tests.helpers import rand_real, rand_spectral, to_dev, to_host

pytestmark = pytest.mark.gpu

# few lines per axis, each length once along y (64 .. 1024) and z (32 .. 512)
FEW = [(16, 64, 32), (16, 128, 64), (16, 256, 128), (16, 512, 256), (16, 1024, 512)]
# more z lines than 8 warps a multiprocessor take
MANY = [(256, 128, 32), (128, 128, 64), (64, 128, 128), (64, 64, 256)]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", FEW + MANY)
def test_warp_line_y_and_z_passes(prec, shape):
    """Plain transforms; then two steps of each solver, the first substep full
    (modes outside the truncation), the others zero-pruned.  Tolerances: the
    rounding of a transform (a few eps log2 n) over 2 steps of order 2."""
    from ghost_b200 import GHOST_COMPLEX_TO_REAL, GHOST_REAL_TO_COMPLEX, Ghost
    box = dict(Lx=1, Ly=1, Lz=0.5, arbsize=True)
    o, ob = Oracle(*shape), Oracle(*shape, **box)
    g = Ghost(*shape, precision=prec)
    cd = g.cdtype_np
    one, tol = (1e-13, 1e-11) if prec == "fp64" else (2e-6, 1e-5)
    r, s = rand_real(o, 5), rand_spectral(o, 6)
    out, real = g.czeros(), g.rzeros()
    g.fftp3d_real_to_complex(g.fftp3d_create_plan(shape, GHOST_REAL_TO_COMPLEX), to_dev(r.astype(g.rdtype_np)), out)
    assert rel_l2(to_host(out), o.fftp3d_real_to_complex(r)) < one
    g.fftp3d_complex_to_real(g.fftp3d_create_plan(shape, GHOST_COMPLEX_TO_REAL), to_dev(s.astype(cd)), real)
    assert rel_l2(to_host(real), o.fftp3d_complex_to_real(s)) < one

    v, a = ([x + 0.01 * rand_spectral(o, k + q) for q, x in enumerate(o.random_solenoidal(k, 1.0, 6.0, 1, amp)[0])]
            for k, amp in ((81, 1.0), (84, 0.3)))
    f = o.random_solenoidal(87, 2.0, 3.0, 0, 1.0)[0]
    th = rand_spectral(o, 88, 0.1)
    dev = lambda q: [to_dev(x.astype(cd)) for x in q]  # noqa: E731
    host = lambda q: [to_host(x) for x in q]  # noqa: E731
    V = dev(v)
    g.hd_run(2, 2, 1e-3, 2e-3, *V)
    assert rel_l2(host(V), o.hd_run(2, 2, 1e-3, 2e-3, v)) <= tol
    V, A = dev(v), dev(a)
    g.mhd_run(2, 2, 1e-3, 1e-3, 2e-3, *V, *A, f=dev(f))
    rv, ra = o.mhd_run(2, 2, 1e-3, 1e-3, 2e-3, v, a, f=f)
    assert rel_l2(host(V), rv) <= tol and rel_l2(host(A), ra) <= tol
    gb = Ghost(*shape, precision=prec, **box)
    V, TH = dev(v), to_dev(th.astype(cd))
    args = (2, 2.5e-4, 5e-4, 5e-4, 0.5, 8.0, 8.0)
    gb.bouss_run(2, *args, *V, TH)
    rv, rt = ob.bouss_run(2, *args, v, th)
    assert rel_l2(host(V) + [to_host(TH)], list(rv) + [rt]) <= tol


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [32, 64, 128])
def test_stresses_through_one_x_pass(prec, n):
    """The six stresses of the closure as spectra: x one by one below 64
    points, in one launch from there on.  The rows are float32, so the error is
    that of six transforms, a sum of three of them and a projection."""
    from ghost_b200 import Ghost
    from ghost_b200.les import LES
    from oracle import les_oracle
    co, gc = Oracle(n), Ghost(n, precision=prec)
    kc = n // 3
    co.set_kmax(float(kc * kc))
    les = LES(gc, kc)
    tau = np.random.default_rng(n).standard_normal((n ** 3, 6)).astype(np.float32)
    F = les.tau_force(to_dev(tau), 0.25)
    ref = les_oracle.tau_force(co, tau.astype(np.float64), 0.25)
    assert rel_l2([to_host(x) for x in F], ref) <= (1e-13 if prec == "fp64" else 2e-6)
