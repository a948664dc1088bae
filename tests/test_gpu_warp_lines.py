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


def _stalled(g, call, kept):
    """call() with every pass's first wait made to run out: GHOST_ERR_TIMEOUT,
    and not a bit of the tensors it would have written."""
    import torch
    from ghost_b200 import GhostError
    before = [x.clone() for x in kept]
    g.set_wait_cap(1000)
    g.inject_stall(True)
    with pytest.raises(GhostError) as err:
        call()
        g.synchronize()
    assert err.value.code == 5
    g.inject_stall(False)
    g.set_wait_cap(0)
    assert all(torch.equal(a, b) for a, b in zip(kept, before))


# every warp-line kernel and size of its groups (one warp per group: nx = 64, FP64)
STALL = [("fp32", (64, 64, 64)), ("fp64", (64, 128, 64)), ("fp32", (128, 256, 128)), ("fp64", (128, 256, 128)),
         ("fp32", (256, 512, 32)), ("fp64", (256, 128, 32)), ("fp32", (1024, 64, 32)), ("fp64", (512, 64, 512)),
         ("fp32", (512, 1024, 32))]


@pytest.mark.parametrize("prec,shape", STALL)
def test_a_wait_that_runs_out_stores_nothing(prec, shape):
    """After a bounded wait ran out, a pass leaves its results unwritten: both
    plain transforms (FP32 512-point x lines, which finish, aside), and steps
    of the three solvers; afterwards the same calls give the bits of a context
    that never saw a timeout."""
    import torch
    from ghost_b200 import GHOST_COMPLEX_TO_REAL, GHOST_REAL_TO_COMPLEX, Ghost
    o = Oracle(*shape)
    g, ref = Ghost(*shape, precision=prec), Ghost(*shape, precision=prec)
    cd = g.cdtype_np
    dev = lambda q: [to_dev(x.astype(cd)) for x in q]  # noqa: E731
    v = dev(o.random_solenoidal(91, 1.0, 6.0, 1, 1.0)[0])
    a = dev(o.random_solenoidal(92, 1.0, 6.0, 1, 0.3)[0])
    th = v[2] * 0.1
    r, s = to_dev(rand_real(o, 93).astype(g.rdtype_np)), to_dev(rand_spectral(o, 94).astype(cd))
    n = shape
    calls = []
    if (prec, shape[0]) != ("fp32", 512):
        def r2c(h, out):
            h.fftp3d_real_to_complex(h.fftp3d_create_plan(n, GHOST_REAL_TO_COMPLEX), r, *out)

        def c2r(h, out):
            h.fftp3d_complex_to_real(h.fftp3d_create_plan(n, GHOST_COMPLEX_TO_REAL), s.clone(), *out)
        calls += [(r2c, [torch.full_like(g.czeros(), 7.0)]), (c2r, [torch.full_like(g.rzeros(), 7.0)])]
    calls += [(lambda h, x: h.hd_run(1, 2, 1e-3, 1e-3, *x), v),
              (lambda h, x: h.bouss_run(1, 2, 2.5e-4, 5e-4, 5e-4, 0.5, 8.0, 8.0, *x), v + [th]),
              (lambda h, x: h.mhd_run(1, 2, 1e-3, 1e-3, 1e-3, *x), v + a)]
    for call, start in calls:
        kept, want = [x.clone() for x in start], [x.clone() for x in start]
        _stalled(g, lambda: call(g, kept), kept)
        call(g, kept)
        call(ref, want)
        g.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(kept, want))


def test_a_wait_that_runs_out_stores_nothing_in_a_closure_or_an_ensemble():
    """The same for a step of an LES with the learned closure (the pass that
    writes its inputs) and for the launches over all classes of an ensemble."""
    import torch
    from ghost_b200 import Ensemble, Ghost, GhostError
    from ghost_b200.les import LES, MLP
    for prec, n in (("fp32", 64), ("fp64", 64), ("fp32", 128)):
        g = Ghost(n, precision=prec)
        v = [g.czeros() for _ in range(3)]
        g.init_random_solenoidal(95, 1.0, n / 3.0, 1, 1.0, *v)
        les = LES(g, n // 3)
        mlp = MLP(0)
        les.set_model("mlp", mlp, grad_scale=0.1, tau_scale=0.02, delta=1.0)
        _stalled(g, lambda: les.run(1, 2, 1e-3, 1e-3, *v), v)
    for prec in ("fp32", "fp64"):
        e = Ensemble([32, 64, 128], [3, 2, 1], precision=prec)
        fields = [e.fields(q) for q in range(3)]
        for q in range(3):
            for x in fields[q]:
                x.copy_(torch.randn(x.shape, dtype=x.real.dtype, device="cuda") * 1e-3)
        torch.cuda.synchronize()
        before = [[x.clone() for x in f] for f in fields]
        for q in range(3):
            e.class_ctx(q).set_wait_cap(1000)
            e.class_ctx(q).inject_stall(True)
        with pytest.raises(GhostError) as err:
            e.run(1, 2, 1e-3)
        assert err.value.code == 5
        assert all(torch.equal(x, y) for f, b in zip(fields, before) for x, y in zip(f, b))
