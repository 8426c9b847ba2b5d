"""GPU tests of the caller's arrays at addresses that the kernels' loads and
stores do not take in place: such arrays go through staging copies, with the
same results as aligned ones."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(built_lib):
    import spectral2d_gb300
    return spectral2d_gb300


def _at(values, offset, mem="pageable"):
    """A copy of the array that starts `offset` bytes past a 64-byte boundary."""
    from spectral2d_gb300.solver import pinned_array
    n = values.nbytes + 128
    raw = pinned_array(n, np.uint8) if mem == "pinned" else np.zeros(n, dtype=np.uint8)
    at = -raw.ctypes.data % 64 + offset
    a = raw[at:at + values.nbytes].view(values.dtype).reshape(values.shape)
    a[...] = values
    assert a.ctypes.data % 64 == offset and a.flags.c_contiguous
    return a


@pytest.mark.parametrize("mem", ["pageable", "pinned"])
@pytest.mark.parametrize("offset", [2, 4, 8, 12])
def test_closure_batches_at_any_address(S, offset, mem):
    """(omega, psi) pairs are loaded 8 bytes at a time; a float array may start
    at any multiple of 4, or (packed buffers) anywhere."""
    from spectral2d_gb300 import _lib as L
    from spectral2d_gb300.solver import _fptr
    rng = np.random.default_rng(offset)
    x = _at(rng.standard_normal((3, 24, 24, 2)).astype(np.float32), 0)
    t = _at(rng.standard_normal((3, 24, 24)).astype(np.float32), 0)
    with S.ClosureNet(24, max_batch=4, seed=1) as net:
        y = net.forward(x)
        loss, g = net.grad(x, t)
        xo, to = _at(x, offset, mem), _at(t, offset, mem)
        assert np.array_equal(net.forward(xo), y)
        for a, b in ((xo, to), (xo, t), (x, to)):
            lo, go = net.grad(a, b)
            assert lo == loss and np.array_equal(go, g)
        yo = _at(np.zeros_like(y), offset, mem)
        L.check(net._L.s2d_cnn_forward_host(net._c, _fptr(x), 3, _fptr(yo)))
        assert np.array_equal(yo, y)


@pytest.mark.parametrize("mem", ["pageable", "pinned", "fresh"])
@pytest.mark.parametrize("n", [24, 96])
def test_state_arrays_at_half_an_element(S, n, mem):
    """The kernels move complex numbers 16 bytes at a time; an array of doubles
    may start 8 bytes off, its pages touched already or not."""
    import oracle as O
    from spectral2d_gb300 import _lib as L
    from spectral2d_gb300.solver import _dptr
    w = O.random_state(O.get_grid_size(n, n), 5, decay=0.1)

    def buf(values=None):
        if mem == "fresh" and values is None:
            raw = np.zeros(2 * w.size + 8)   # pages not touched yet
            at = (-raw.ctypes.data % 16) // 8 + 1
            a = raw[at:at + 2 * w.size].view(np.complex128).reshape(w.shape)
        else:
            a = _at(np.full_like(w, np.nan) if values is None else values, 8, "pinned" if mem == "pinned" else "pageable")
        assert a.ctypes.data % 16 == 8
        return a

    shape = w.shape[::-1]
    with S.Spectral2D(n, nu=0.01) as r:
        r.set_state(w)
        dW = r.compute_rhs()
        r.integrate_one_step(1e-3)
        w1, p1 = r.get_state()
    with S.Spectral2D(n, nu=0.01) as s:
        s.set_state(buf(w))
        d = buf()
        L.check(s._L.s2d_compute_rhs(s._h, _dptr(d.view(np.float64)), *shape))
        gw, gp = buf(w), buf()
        s.integrate_one_step_host(gw, 1e-3, gp, inplace=True)
        hw, hp = buf(), np.full_like(w, np.nan)   # one staged, one in place
        L.check(s._L.s2d_get_state(s._h, _dptr(hw.view(np.float64)), _dptr(hp.view(np.float64)), *shape))
    assert np.array_equal(d, dW)
    for a, b in ((gw, w1), (gp, p1), (hw, w1), (hp, p1)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("mem", ["pageable", "pinned", "fresh"])
def test_closure_batches_through_staging_copies(S, mem, monkeypatch):
    """S2D_HOST_IO=copy: a batch smaller than the network's through the staging
    buffer and the copy-out, bit for bit what arrays in place give; and (without
    it) an input whose pages are not resident, staged beside one in place."""
    from spectral2d_gb300 import _lib as L
    from spectral2d_gb300.solver import _fptr
    rng = np.random.default_rng(3)
    x = rng.standard_normal((3, 24, 24, 2)).astype(np.float32)
    t = rng.standard_normal((3, 24, 24)).astype(np.float32)
    if mem == "fresh":
        x = np.zeros_like(x)
    out = []
    for io in ("in_place", "copy"):
        if io == "copy":
            monkeypatch.setenv("S2D_HOST_IO", "copy")
        with S.ClosureNet(24, max_batch=5, seed=1) as net:
            net.set_scales([2.0, 0.5, 0.25])
            xs = np.zeros(x.shape, np.float32) if mem == "fresh" else _at(x, 0, mem)
            loss, g = net.grad(xs, _at(t, 0, "pageable" if mem == "fresh" else mem))
            y = _at(np.full_like(t, np.nan), 0, "pinned" if mem == "pinned" else "pageable")
            L.check(net._L.s2d_cnn_forward_host(net._c, _fptr(xs), 3, _fptr(y)))
            out.append((loss, g, y.copy()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
