"""GPU: the maps' workspace: passes and copies of mu at the limits of what fits, and volumes that do not start on
16 bytes.  The copies, the pass size and the width of the loads move data, never results."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _volumes(n, s, offset=0):
    g = torch.Generator(device="cuda").manual_seed(n)
    buf = [torch.rand(s * n * n + offset, device="cuda", generator=g) * 0.02 for _ in range(2)]
    return [b[offset:].view(s, n, n) for b in buf]


def _scans(call):
    """Result of call and the number of column scans that it launched (None where the profiler sees no
    kernels)."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out = call()
        torch.cuda.synchronize()
    counts = {e.key: e.count for e in prof.key_averages() if "maps_" in e.key}
    return out, sum(v for k, v in counts.items() if "maps_scan_kernel" in k) if counts else None


@pytest.mark.parametrize("n", [64, 33, 130])
@pytest.mark.parametrize("n_ang,quads", [(1, False), (3, False), (40, False), (40, True)])
def test_maps_passes_and_copies(n, n_ang, quads):
    """The workspace that compute_maps takes by itself holds the copies and every entry of a small set: one
    pass; last_passes names the passes of any workspace; results do not depend on it."""
    from pycorrectedemissionct_b200 import core

    s = 2
    mu_in, mu_out = _volumes(n, s)
    if quads:
        mu_out = mu_in
    rad32 = np.linspace(0, 2 * np.pi, n_ang, endpoint=False).astype(np.float32)
    args = (mu_in, mu_out, rad32)
    ref, scans = _scans(lambda: core.compute_maps(*args))
    assert core.compute_maps.last_passes == 1 and scans in (1, None)
    need = core.maps_entry_bytes(n, s)
    copies = 2 * core._maps_copy_bytes(n, s)  # (sides of 33 and 64 with few angles take none)
    # one entry in place (narrow loads where n % 4 != 0), one and three beside the copies, and between
    for nbytes in (need, need + copies // 2, need + copies, 3 * need + copies - 4, 3 * need + copies):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        got, scans = _scans(lambda: core.compute_maps(*args, workspace=ws))
        assert scans in (core.compute_maps.last_passes, None)
        assert torch.equal(got, ref)


@pytest.mark.parametrize("n", [64, 33])
def test_maps_of_volumes_off_alignment(n):
    """Volumes that begin 4 bytes past a 16-byte boundary, with and without room for the copies."""
    from pycorrectedemissionct_b200 import core

    s = 3
    rad32 = np.linspace(0, 2 * np.pi, 9, endpoint=False).astype(np.float32)
    mu_in, mu_out = _volumes(n, s, 1)
    assert mu_in.data_ptr() % 16 == 4
    ref = core.compute_maps(mu_in.clone(), mu_out.clone(), rad32)
    assert torch.equal(core.compute_maps(mu_in, mu_out, rad32), ref)
    ws = torch.empty(core.maps_entry_bytes(n, s), dtype=torch.uint8, device="cuda")
    assert torch.equal(core.compute_maps(mu_in, mu_out, rad32, workspace=ws), ref)
