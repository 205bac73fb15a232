"""GPU: the back projection at the edges of its tiles, line segments and cluster rule, against the
FP64 oracle: line counts around the segment counts' steps (16, 32, 64 lines) and the chunk of 16,
sides around the tiles (32, 64) and the tile-height rule (192), angles whose detector edges fall
exactly on pixels (0, 90 degrees), several detectors, and batches on both sides of the cluster rule
(equal bits)."""

import numpy as np
import pytest

from conftest import rel_l2, report

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-5  # FP32 sums of at most a few hundred lines against FP64


@pytest.mark.parametrize("n,n_ang,n_det", [(2, 4, 1), (3, 15, 1), (31, 16, 1), (32, 17, 1), (33, 31, 1), (64, 32, 1),
                                           (65, 63, 1), (96, 64, 1), (192, 65, 1), (193, 40, 2), (200, 360, 1)])
def test_bp_matches_port_and_batches_agree(n, n_ang, n_det):
    from oracle import port
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    angles = np.linspace(0, 2 * np.pi, n_ang, endpoint=False)
    rng = np.random.default_rng(n + n_ang)
    # enough slices that the large batch is past the cluster rule for every side
    s = 352 // max(1, -(-n // 32) * -(-n // (64 if n > 192 else 32))) + 1
    y = torch.from_numpy(rng.uniform(0.5, 1.5, size=(s, n_det, n_ang, n)).astype(np.float32)).to(dev)
    maps = torch.from_numpy(rng.uniform(0.3, 1.0, size=(1, n_ang, n_det, n, n)).astype(np.float32)).to(dev)
    c = core.XrfCore(n, angles, n_det=n_det, device=dev)
    one = c.bp(y[:1])
    assert torch.equal(c.bp(y)[:1], one)
    sym = c.bp(y[:1], "symmetric", maps)
    assert torch.equal(c.bp(y, "symmetric", maps.expand(s, -1, -1, -1, -1).contiguous())[:1], sym)
    _, deg32 = port.backend_angles(angles)
    y64, m64 = y[0].double().cpu().numpy(), maps[0].double().cpu().numpy()
    e = rel_l2(one[0].cpu().numpy(), port.bp_xrf(y64, m64, deg32))
    es = rel_l2(sym[0].cpu().numpy(), port.bp_xrf(y64, m64, deg32, is_symmetric=True))
    report(f"bp n={n} lines={n_ang * n_det}", e, TOL)
    assert e < TOL and es < TOL


@pytest.mark.parametrize("n_ang", [1, 16, 70])
@pytest.mark.parametrize("n", [2, 3, 33, 64, 193])
def test_bp_takes_the_last_bin_itself(n, n_ang):
    """Lines at angle 0, whose last image column lies exactly on the last detector bin: np.interp returns that
    bin, whatever its neighbour holds (3e7 beside 0.5 here, or infinity).  Every pixel is exactly on a bin
    and every sum is exact in FP32, so the results are equal, for a batch on either side of the
    cluster rule, in the reference and the symmetric mode."""
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    s = 352 // max(1, -(-n // 32) * -(-n // (64 if n > 192 else 32))) + 1
    y = np.ones((1, n_ang, n), dtype=np.float32)
    y[..., -2], y[..., -1] = 3e7, 0.5
    c = core.XrfCore(n, np.zeros(n_ang), device=dev)
    maps = torch.ones((s, n_ang, 1, n, n), device=dev)
    t = np.arange(n) - n // 2
    ref = n_ang * np.interp(t, t, y[0, 0].astype(np.float64), left=0, right=0)
    yd = torch.from_numpy(y).to(dev).expand(s, -1, -1, -1).contiguous()
    for slices in (1, s):
        for args in (("reference",), ("symmetric", maps[:slices])):
            got = c.bp(yd[:slices], *args).double().cpu().numpy()
            assert np.array_equal(got, np.broadcast_to(ref, got.shape))
    yd[..., -2] = float("inf")
    assert torch.equal(c.bp(yd)[..., -1], torch.full((s, n), 0.5 * n_ang, device=dev))


@pytest.mark.parametrize("n", [33, 130, 251])
def test_bp_interpolates_edge_pixels_in_double(n):
    """Pixels within 0.01 bin inside the last detector bin, on a line that rises from -1 to 0 there: the value is
    the distance to the edge itself, known to 1e-11 and rounded to FP32 once (formed in FP32 as
    -1 + (1 + d) it would be off by up to 6e-8)."""
    from oracle import port
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    y = np.zeros((1, 1, 1, n), dtype=np.float32)
    y[..., -2] = -1.0
    jj, ii = np.meshgrid(np.arange(n) - n // 2, np.arange(n) - n // 2)
    checked = 0
    for angle in np.random.default_rng(n).uniform(0, 2 * np.pi, 60):
        _, deg32 = port.backend_angles(np.array([angle]))
        rad = np.deg2rad(deg32[0])
        d = (n - 1 - n // 2) - (jj * np.cos(rad).astype(np.float64) - ii * np.sin(rad).astype(np.float64))
        near = (d > 0) & (d < 0.009)
        got = core.XrfCore(n, [angle], device=dev).bp(torch.from_numpy(y).to(dev))[0].double().cpu().numpy()
        assert np.all(np.abs(got + d)[near] <= 1e-11 + 2.0**-24 * d[near])
        checked += int(near.sum())
    assert checked > 0


@pytest.mark.parametrize("n_ang", [1, 16])
@pytest.mark.parametrize("n", [33, 64])
def test_symmetric_bp_of_unbounded_maps_at_the_edges(n, n_ang):
    """A map value of infinity makes its pixel infinite, on the detector's edge bins (angle 0: the first and last
    columns) as inside."""
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    c = core.XrfCore(n, np.zeros(n_ang), device=dev)
    y = torch.ones((1, 1, n_ang, n), device=dev)
    maps = torch.ones((1, n_ang, 1, n, n), device=dev)
    want = torch.full((1, n, n), float(n_ang), device=dev)
    for i, j in ((0, 0), (1, n - 1), (n // 2, n // 3), (n - 1, n - 1)):
        maps[0, n_ang // 2, 0, i, j] = want[0, i, j] = float("inf")
    assert torch.equal(c.bp(y, "symmetric", maps), want)


@pytest.mark.parametrize("n_ang", [4, 20, 70])
@pytest.mark.parametrize("n", [31, 33, 64, 96, 130, 192, 200])
def test_bp_tile_rows_and_clusters_give_the_same_bits(n, n_ang):
    """Tiles of 32 and of 64 rows, in clusters and not: batches on all sides of both rules hold the slice of a
    batch of one, in the reference and the symmetric mode."""
    from pycorrectedemissionct_b200 import core

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    tiles32, tiles64 = ((n + 31) // 32) ** 2, (n + 31) // 32 * ((n + 63) // 64)
    segs = 8 if n_ang >= 64 else 2 if n_ang >= 16 else 1
    few = (296 if segs > 1 else 592) // segs // tiles32  # the last batch of 32-row tiles
    batches = sorted({1, few, few + 1, 351 // tiles64, 352 // tiles64 + 1} - {0})
    g = torch.Generator(device=dev).manual_seed(n * n_ang)
    y = torch.rand((batches[-1], 1, n_ang, n), device=dev, generator=g)
    maps = torch.rand((1, n_ang, 1, n, n), device=dev, generator=g).expand(batches[-1], -1, -1, -1, -1).contiguous()
    c = core.XrfCore(n, np.linspace(0, 2 * np.pi, n_ang, endpoint=False), device=dev)
    ref, sym = c.bp(y[:1]), c.bp(y[:1], "symmetric", maps[:1])
    for s in batches[1:]:
        assert torch.equal(c.bp(y[:s])[:1], ref) and torch.equal(c.bp(y[:s].flip(0).contiguous())[-1:], ref)
        assert torch.equal(c.bp(y[:s], "symmetric", maps[:s])[:1], sym)
