"""The passes over point pairs that screen in FP32, where FP32 itself gives out: coordinates
whose squared distances exceed it or fall below its normal numbers, and scales outside
its range. The FP64 values decide, bit for bit (sums of squares in the order of the
dimensions, rounded after every operation)."""
import pytest

from pdot import _abi

pytestmark = pytest.mark.gpu

# magnitude of the coordinates, and the scale that brings a squared distance to about one
MAGNITUDES = [(1.0, 1.0), (1e18, 1e-36), (1e19, 1e-38), (3e19, 1e-39), (1e20, 1e-40), (3e22, 1e-45), (1e25, 1e-50),
              (1e37, 1e-74), (1e-10, 1e20), (1e-19, 1e38), (1e-22, 1e44), (1e-30, 1e60)]


def _points(torch, count, dim, magnitude, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(count, dim, generator=g, device="cuda", dtype=torch.float64) * magnitude
    return x.float()


def _sqdist(torch, x, y):
    d = torch.zeros(x.shape[0], y.shape[0], device="cuda", dtype=torch.float64)
    for k in range(x.shape[1]):
        e = x[:, k].double()[:, None] - y[:, k].double()[None, :]
        d += e * e
    return d


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("magnitude,scale", MAGNITUDES)
def test_c_transform_at_the_ends_of_fp32(cuda, magnitude, scale, dim):
    import torch

    lib = _abi.load()
    n, centres = 700, 3001
    p = _points(torch, n, dim, magnitude, 1)
    c = _points(torch, centres, dim, magnitude, 2).double()
    v = torch.randn(centres, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(3))
    for s, dual in ((scale, 1.0), (scale, 0.01), (-scale, 1.0), (0.0, 1.0)):
        out = torch.empty(n, device="cuda", dtype=torch.float64)
        w = v * dual
        rc = lib.pdot_points_c_transform(n, centres, dim, p.data_ptr(), c.data_ptr(), w.data_ptr(), s, out.data_ptr(), None)
        _abi.check(lib, rc, "pdot_points_c_transform")
        want = (s * _sqdist(torch, p, c) - w[None, :]).min(1).values
        assert torch.equal(out, want), (s, dual)


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("magnitude", [m for m, _ in MAGNITUDES])
def test_largest_distance_at_the_ends_of_fp32(cuda, magnitude, dim):
    import torch

    lib = _abi.load()
    m, n = 2300, 2100  # above the size from which the cost builder screens
    x, y = _points(torch, m, dim, magnitude, 4), _points(torch, n, dim, magnitude, 5)
    want = _sqdist(torch, x, y).max()
    out = torch.empty(1, device="cuda", dtype=torch.float64)
    _abi.check(lib, lib.pdot_points_max_sqdist(m, n, dim, x.data_ptr(), y.data_ptr(), out.data_ptr(), None), "max")
    assert torch.equal(out[0], want)
    x64, y64 = x.double(), y.double()
    cost = torch.empty(n, m, device="cuda", dtype=torch.float64)  # column-major m x n
    _abi.check(lib, lib.pdot_sqeuclid_cost_f64(m, n, dim, x64.data_ptr(), y64.data_ptr(), 1, cost.data_ptr(), None), "cost")
    assert torch.equal(cost.T, _sqdist(torch, x, y) / want)


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("shift", [0.5, 1e3, 1e6])
def test_c_transform_of_points_far_from_the_origin(cuda, shift, dim):
    """Points of a unit cube at a distance, whose coordinates FP32 holds to fewer digits."""
    import torch

    lib = _abi.load()
    n, centres = 1000, 2000
    p = (_points(torch, n, dim, 1.0, 6).double() + shift).float()
    c = _points(torch, centres, dim, 1.0, 7).double() + shift
    v = torch.randn(centres, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(8))
    for dual in (0.0, 0.1):
        out = torch.empty(n, device="cuda", dtype=torch.float64)
        w = v * dual
        rc = lib.pdot_points_c_transform(n, centres, dim, p.data_ptr(), c.data_ptr(), w.data_ptr(), 1.0, out.data_ptr(), None)
        _abi.check(lib, rc, "pdot_points_c_transform")
        d = torch.zeros(n, centres, device="cuda", dtype=torch.float64)
        for k in range(dim):
            e = p[:, k].double()[:, None] - c[None, :, k]
            d += e * e
        assert torch.equal(out, (d - w[None, :]).min(1).values)


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("second", [1, 31, 128, 129, 160, 161, 192, 193, 256, 257])
def test_pair_passes_over_few_points(cuda, second, dim):
    """Both sides of the size up to which the second set is one tile in FP64."""
    import torch

    lib = _abi.load()
    for first in (1, 255, 257, 3000):
        x, y = _points(torch, first, dim, 1.0, 9), _points(torch, second, dim, 1.0, 10)
        d = _sqdist(torch, x, y)
        top = torch.empty(1, device="cuda", dtype=torch.float64)
        _abi.check(lib, lib.pdot_points_max_sqdist(first, second, dim, x.data_ptr(), y.data_ptr(), top.data_ptr(), None), "max")
        assert torch.equal(top[0], d.max())
        c = y.double()
        v = torch.randn(second, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(11))
        out = torch.empty(first, device="cuda", dtype=torch.float64)
        rc = lib.pdot_points_c_transform(first, second, dim, x.data_ptr(), c.data_ptr(), v.data_ptr(), 1.5, out.data_ptr(), None)
        _abi.check(lib, rc, "pdot_points_c_transform")
        assert torch.equal(out, (1.5 * d - v[None, :]).min(1).values)


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("kind", ["zero", "smooth", "flat", "own", "twins"])
def test_c_transform_where_many_centres_nearly_tie(cuda, kind, dim):
    """Duals under which centres differ by less than FP32 tells apart: none, a smooth potential, one that
    makes every centre as good as the next, centres that are the points, and centres that coincide."""
    import torch

    lib = _abi.load()
    n, centres = 1500, 2500
    p = _points(torch, n, dim, 1.0, 12)
    c = _points(torch, centres, dim, 1.0, 13).double()
    v = torch.zeros(centres, device="cuda", dtype=torch.float64)
    if kind == "smooth":
        v = 0.3 * (c * c).sum(1) + 0.1 * c[:, 0]
    elif kind == "flat":  # |x - c|^2 - |c|^2 hardly depends on c for points near the origin
        v = (c * c).sum(1)
        p = p * 1e-6
    elif kind == "own":
        c[:n] = p.double()
    elif kind == "twins":
        c[1000:] = c[torch.arange(1000, centres, device="cuda") % 7]
    for scale in (1.0, 0.37, -1.0):
        w = scale * v
        out = torch.empty(n, device="cuda", dtype=torch.float64)
        rc = lib.pdot_points_c_transform(n, centres, dim, p.data_ptr(), c.data_ptr(), w.data_ptr(), scale, out.data_ptr(), None)
        _abi.check(lib, rc, "pdot_points_c_transform")
        d = torch.zeros(n, centres, device="cuda", dtype=torch.float64)
        for k in range(dim):
            e = p[:, k].double()[:, None] - c[None, :, k]
            d += e * e
        assert torch.equal(out, (scale * d - w[None, :]).min(1).values), scale


@pytest.mark.parametrize("dim", [1, 2, 3, 4, 5, 6, 9])
@pytest.mark.parametrize("m,n", [(1, 1), (1, 4000), (3000, 1), (2, 300), (63, 500), (64, 500), (65, 33), (513, 260), (1000, 16),
                                 (400, 400), (401, 400), (402, 400)])
def test_cost_of_few_rows_and_of_more_dimensions(cuda, m, n, dim):
    """Both sides of the number of rows up to which a thread takes an entry, and dimensions beyond those
    that are compiled in; as given and normalised."""
    import torch

    lib = _abi.load()
    x, y = _points(torch, m, dim, 1.0, 14).double(), _points(torch, n, dim, 1.0, 15).double()
    d = _sqdist(torch, x, y)
    for normalise in (0, 1):
        cost = torch.full((n * m + 1,), 7.0, device="cuda", dtype=torch.float64)
        rc = lib.pdot_sqeuclid_cost_f64(m, n, dim, x.data_ptr(), y.data_ptr(), normalise, cost.data_ptr(), None)
        _abi.check(lib, rc, "pdot_sqeuclid_cost_f64")
        assert torch.equal(cost[:-1].view(n, m).T, d / d.max() if normalise else d)
        assert cost[-1] == 7.0
