"""The plain 512-point FP32 x transforms with one warp per line
(fftp3d_real_to_complex / fftp3d_complex_to_real) against the oracle, and
the bounded-wait timeout path of their TMA rings."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from tests.conftest import rel_l2
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu

def ghost(*shape, **kw):
    from ghost_b200 import Ghost
    return Ghost(*shape, **kw)


@pytest.mark.parametrize("shape", [(512, 16, 32), (512, 32, 16)])
def test_plain_r2c_warp_lines(shape):
    """fftp3d_real_to_complex at nx = 512 (FP32) runs the warp-line x pass."""
    from ghost_b200 import GHOST_REAL_TO_COMPLEX
    from tests.helpers import rand_real
    o = Oracle(*shape)
    g = ghost(*shape, precision="fp32")
    r = rand_real(o, 5)
    ref = o.fftp3d_real_to_complex(r)
    plan = g.fftp3d_create_plan(shape, GHOST_REAL_TO_COMPLEX)
    out = g.czeros()
    g.fftp3d_real_to_complex(plan, to_dev(r.astype(np.float32)), out)
    assert rel_l2(to_host(out), ref) < 2e-6


@pytest.mark.parametrize("shape", [(512, 16, 32), (512, 32, 16)])
def test_plain_c2r_warp_lines(shape):
    """fftp3d_complex_to_real at nx = 512 (FP32), a non-Hermitian input
    (only the real parts of the kx = 0 and Nyquist values count)."""
    from ghost_b200 import GHOST_COMPLEX_TO_REAL
    from tests.helpers import rand_spectral
    o = Oracle(*shape)
    g = ghost(*shape, precision="fp32")
    c = rand_spectral(o, 6)
    ref = o.fftp3d_complex_to_real(c)
    plan = g.fftp3d_create_plan(shape, GHOST_COMPLEX_TO_REAL)
    cin = to_dev(c.astype(np.complex64))
    keep = cin.clone()
    out = g.rzeros()
    g.fftp3d_complex_to_real(plan, cin, out)
    assert rel_l2(to_host(out), ref) < 2e-6
    assert bool((cin == keep).all())


LINES = [("fp32", n) for n in (32, 64, 128, 256, 1024)] + [("fp64", n) for n in (32, 64, 128, 256, 512, 1024)]


@pytest.mark.parametrize("prec,nx", LINES)
def test_plain_lines_of_every_length(prec, nx):
    """Both plain transforms at every other line length, on non-cubic grids
    with one and with several tiles per y, against the oracle."""
    from ghost_b200 import GHOST_COMPLEX_TO_REAL, GHOST_REAL_TO_COMPLEX
    from tests.helpers import rand_real, rand_spectral
    for ny, nz in ((16, 16), (32, 64)):
        o = Oracle(nx, ny, nz)
        g = ghost(nx, ny, nz, precision=prec)
        tol = 1e-13 if prec == "fp64" else 2e-6
        r, c = rand_real(o, 5), rand_spectral(o, 6)
        fwd = g.fftp3d_create_plan((nx, ny, nz), GHOST_REAL_TO_COMPLEX)
        inv = g.fftp3d_create_plan((nx, ny, nz), GHOST_COMPLEX_TO_REAL)
        out, real = g.czeros(), g.rzeros()
        g.fftp3d_real_to_complex(fwd, to_dev(r.astype(g.rdtype_np)), out)
        assert rel_l2(to_host(out), o.fftp3d_real_to_complex(r)) < tol
        g.fftp3d_complex_to_real(inv, to_dev(c.astype(g.cdtype_np)), real)
        assert rel_l2(to_host(real), o.fftp3d_complex_to_real(c)) < tol


def test_plain_timeout_reports_and_recovers():
    """With the stall injected the warp-line transforms record
    GHOST_ERR_TIMEOUT and finish; the context then works normally."""
    from ghost_b200 import GHOST_REAL_TO_COMPLEX, GhostError
    from tests.helpers import rand_real
    shape = (512, 16, 16)
    o = Oracle(*shape)
    g = ghost(*shape, precision="fp32")
    r = rand_real(o, 7)
    plan = g.fftp3d_create_plan(shape, GHOST_REAL_TO_COMPLEX)
    out = g.czeros()
    g.set_wait_cap(1000)
    g.inject_stall(True)
    g.fftp3d_real_to_complex(plan, to_dev(r.astype(np.float32)), out)
    with pytest.raises(GhostError) as err:
        g.synchronize()
    assert err.value.code == 5
    g.inject_stall(False)
    g.set_wait_cap(0)
    g.fftp3d_real_to_complex(plan, to_dev(r.astype(np.float32)), out)
    g.synchronize()
    assert rel_l2(to_host(out), o.fftp3d_real_to_complex(r)) < 2e-6
