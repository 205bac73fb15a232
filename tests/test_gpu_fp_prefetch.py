"""Forward projection with the next chunk's map rows asked for ahead: rows of any alignment and width."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,first", [(65, 1), (66, 0), (129, 1), (130, 3), (132, 1), (257, 2)])
def test_fp_with_maps_at_odd_rows_equals_fp_of_the_product(n, first, dtype):
    """One detector, unit weights: fp(x, map) of one angle is fp(x * map) of that angle, bit for bit (the
    staged product is the same FP32 product), for sizes with a second chunk, rows that are not whole
    16-byte units and maps that begin at any element of their buffer."""
    from pycorrectedemissionct_b200 import core

    a = 9
    c = core.XrfCore(n, np.linspace(0.1, 2 * np.pi, a))
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand((1, n, n), device="cuda", generator=g)
    buf = (torch.rand(first + a * n * n, device="cuda", generator=g) + 0.5).to(dtype)
    maps = buf[first:].view(1, a, 1, n, n)
    sino = c.fp(x, maps)
    for k in range(a):
        one = core.XrfCore(n, np.linspace(0.1, 2 * np.pi, a)[k : k + 1])
        assert torch.equal(sino[:, :, k], one.fp(x * maps[:, k, 0].float())[:, :, 0])


@pytest.mark.parametrize("n,channels", [(3, 1), (65, 2), (132, 3), (257, 2), (512, 2)])
def test_fields_fill_leaves_out_only_unread_quads(n, channels):
    """Fields against the two-slice kernel, which stages by row ranges: the same sums, bit for bit."""
    from pycorrectedemissionct_b200 import _lib, core

    a, d = 11, 2
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand((channels, n, n), device="cuda", generator=g)
    fields = torch.rand((1, a, d + 1, n, n), device="cuda", generator=g)
    out = []
    for variant in (0, _lib.CCT_VARIANT_FP_SLICES2):
        c = core.XrfCore(n, np.linspace(0.0, 2 * np.pi, a), n_det=d, variant=variant)
        c.set_channels(np.linspace(0.5, 1.5, channels))
        # what the chunk before left in the box must not show: a second pass over another volume
        c.fp(torch.full_like(x, 1e30), fields)
        out.append(c.fp(x, fields))
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("n,channels", [(2, 2), (3, 2), (3, 4), (5, 2)])
def test_fields_fill_of_the_smallest_sides(n, channels):
    """The same with two channels at least: the two-slice kernel takes pairs only, and one slice goes to the
    plain kernel itself."""
    test_fields_fill_leaves_out_only_unread_quads(n, channels)
