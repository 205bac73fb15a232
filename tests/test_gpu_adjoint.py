"""GPU: the exact adjoint at the edges of its kernel (64 pixels per CTA, lines in chunks of 32, four threads
per pixel) against the scatter definition in FP64, with and without maps, for odd sides and several
detectors."""

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-5  # FP32 sample positions against FP64


@pytest.mark.parametrize("n,n_ang,n_det", [(2, 3, 1), (8, 1, 1), (9, 32, 1), (33, 33, 2), (64, 5, 1), (71, 65, 1)])
def test_adjoint_matches_port(n, n_ang, n_det):
    from oracle import port
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(n * n_ang)
    angles = np.linspace(0, 2 * np.pi, n_ang, endpoint=False) + (0.0 if n_ang > 1 else 0.3)
    c = core.XrfCore(n, angles, n_det=n_det, device=dev)
    _, deg32 = port.backend_angles(angles)
    y = rng.uniform(0.5, 1.5, size=(2, n_det, n_ang, n)).astype(np.float32)
    maps = rng.uniform(0.3, 1.0, size=(2, n_ang, n_det, n, n)).astype(np.float32)
    got = c.bp(torch.from_numpy(y).to(dev), "adjoint", torch.from_numpy(maps).to(dev)).double().cpu().numpy()
    for s in range(2):
        ref = port.fp_xrf_adjoint(y[s].astype(np.float64), maps[s].astype(np.float64), deg32, n)
        assert rel_l2(got[s], ref) < TOL
    if n_det == 1:
        got = c.bp(torch.from_numpy(y).to(dev), "adjoint").double().cpu().numpy()
        assert rel_l2(got[1], port.fp_xrf_adjoint(y[1, 0].astype(np.float64), None, deg32, n)) < TOL


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("n,angle", [(9, 0.0), (33, 0.3), (33, np.pi / 4), (64, 2.0), (71, np.pi / 2)])
def test_adjoint_keeps_a_bad_bin_to_its_pixels(n, angle, bad):
    """A bin that is not finite reaches the pixels that a bin of 1 reaches, and no others (candidates past
    the reach of the hats, or on lattice rows outside the image, add nothing)."""
    from oracle import port
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    c = core.XrfCore(n, [angle], device=dev)
    _, deg32 = port.backend_angles(np.array([angle]))
    for k in (0, 1, n // 2, n - 1):
        y = torch.zeros((1, 1, 1, n), device=dev)
        y[..., k] = 1.0
        one = c.bp(y, "adjoint")
        ref = port.fp_xrf_adjoint(y[0, 0].double().cpu().numpy(), None, deg32, n)
        assert np.abs(one[0].double().cpu().numpy() - ref).max() < 1e-4
        y[..., k] = bad
        assert torch.equal(torch.isfinite(c.bp(y, "adjoint")), one == 0.0)


@pytest.mark.parametrize("n,angle", [(9, 0.2), (33, 0.9), (64, 2.0), (71, 3.5)])
def test_adjoint_forms_hat_products_in_double(n, angle):
    """One bin of 1: a pixel is the sum of the products of its samples' FP32 hats, formed in FP64 and rounded to
    FP32 once; the FP32 positions are mirrored here, so the results are equal."""
    from oracle import port
    from test_host import _fma32
    from pycorrectedemissionct_b200 import core, geometry

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    f = np.float32
    _, deg32 = port.backend_angles(np.array([angle]))
    m00, m01, m02, m10, m11, m12 = geometry.fp_matrices(deg32, n)[0]
    c = core.XrfCore(n, [angle], device=dev)
    r, axis = np.arange(n, dtype=f)[:, None], np.arange(n, dtype=f)[None, :]
    for k in (0, n // 2, n - 1):
        y = torch.zeros((1, 1, 1, n), device=dev)
        y[..., k] = 1.0
        hx = np.maximum(f(1) - np.abs(_fma32(m01, r, _fma32(m00, f(k), m02)) - axis), f(0)).astype(np.float64)
        hy = np.maximum(f(1) - np.abs(_fma32(m11, r, _fma32(m10, f(k), m12)) - axis), f(0)).astype(np.float64)
        want = (hy.T @ hx).astype(f)
        assert np.array_equal(c.bp(y, "adjoint")[0].cpu().numpy(), want)


@pytest.mark.parametrize("n,n_ang,s", [(33, 1, 31), (33, 3, 31), (64, 3, 8), (33, 4, 208), (33, 4, 209), (64, 37, 57), (130, 5, 14)])
def test_adjoint_with_one_thread_per_pixel(n, n_ang, s):
    """Batches on both sides of the rule for the threads of a pixel: the first and the last slice against the
    scatter definition in FP64."""
    from oracle import port
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    angles = np.linspace(0.2, 2 * np.pi, n_ang, endpoint=False)
    g = torch.Generator(device=dev).manual_seed(n * s)
    y = torch.rand((s, 1, n_ang, n), device=dev, generator=g) + 0.5
    maps = torch.rand((1, n_ang, 1, n, n), device=dev, generator=g).expand(s, -1, -1, -1, -1).contiguous()
    got = core.XrfCore(n, angles, device=dev).bp(y, "adjoint", maps).double().cpu().numpy()
    _, deg32 = port.backend_angles(angles)
    for k in (0, s - 1):
        ref = port.fp_xrf_adjoint(y[k].double().cpu().numpy(), maps[k].double().cpu().numpy(), deg32, n)
        assert rel_l2(got[k], ref) < TOL
