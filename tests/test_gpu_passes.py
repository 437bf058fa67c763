"""The device passes beside a solve at the sizes where they can go wrong: tiles and
chunks that end inside a column or a row, the smallest sizes, unaligned buffers, and
values that leave the range their fast paths take.

Tolerances: the cost builder and the two passes over point pairs give the FP64 result
bit for bit (products and sums of each entry in one order, and a maximum or minimum has
no order). The rounded plan's entries are sums of at most m + n terms in another order,
64-bit: 1e-12 relative, as for the host entry."""
import numpy as np
import oracle
import pytest

from pdot import _abi, instances, multiscale

pytestmark = pytest.mark.gpu


def _cost(x, y, normalise=True):
    C = np.zeros((x.shape[0], y.shape[0]))
    for k in range(x.shape[1]):
        C += (x[:, k : k + 1] - y[None, :, k]) ** 2
    with np.errstate(invalid="ignore"):
        mx = np.fmax.reduce(C, axis=None, initial=0.0)
        return C / mx if normalise and mx > 0 else C


def _device_cost(cuda, x, y, normalise, shift=0):
    import torch

    (m, d), n = x.shape, y.shape[0]
    lib = _abi.load()
    dx, dy = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    buf = torch.full((m * n + shift,), -1.0, dtype=torch.float64, device=cuda)
    _abi.check(lib, lib.pdot_sqeuclid_cost_f64(m, n, d, dx.data_ptr(), dy.data_ptr(), normalise,
                                               buf.data_ptr() + 8 * shift, None), "pdot_sqeuclid_cost_f64")
    torch.cuda.synchronize()
    return buf[shift:].cpu().numpy().reshape(n, m).T


@pytest.mark.parametrize("normalise", [0, 1])
@pytest.mark.parametrize("m,n,d", [(1, 1, 1), (2, 1, 2), (3, 2, 3), (512, 17, 4), (513, 300, 2), (1026, 33, 5), (2047, 1, 7)])
def test_cost_builder_is_exact(cuda, m, n, d, normalise):
    rng = np.random.default_rng(m + n)
    x, y = rng.normal(size=(m, d)), rng.normal(size=(n, d))
    for shift in (0, 1):
        assert np.array_equal(_device_cost(cuda, x, y, normalise, shift), _cost(x, y, normalise))


@pytest.mark.parametrize("scale", [0.0, 1e-160, 1e-90, 1e90, 1e150, 1e154])
def test_cost_builder_is_exact_at_the_ends_of_the_range(cuda, scale):
    """All points equal, squares below and above the range of the fast quotient, and infinities."""
    rng = np.random.default_rng(5)
    x, y = scale * rng.uniform(1, 2, (70, 2)), scale * rng.uniform(-2, -1, (41, 2))
    x[3], y[4] = 0.0, 0.0
    with np.errstate(over="ignore", invalid="ignore"):
        want = _cost(x, y)
        np.testing.assert_array_equal(_device_cost(cuda, x, y, 1), want)
        x[5, 1] = np.nan
        want = _cost(x, y)
    np.testing.assert_array_equal(_device_cost(cuda, x, y, 1), want)


@pytest.mark.parametrize("offset,spread", [(0.0, 1.0), (1e4, 1e-3), (0.0, 1e-25), (0.0, 1e25), (-1e30, 1e16), (0.0, 1e45)])
@pytest.mark.parametrize("m,n,d", [(700, 1030, 3), (1, 4200001, 1), (513, 8300, 2), (2300, 1930, 3), (2047, 2051, 4)])
def test_cost_maximum_is_exact(cuda, m, n, d, offset, spread):
    """Bit for bit on both sides of 2^22 pairs, where FP32 tells the pairs apart and where it does not, and
    with a first point that is not a number or infinite."""
    rng = np.random.default_rng(m + n + d)
    x, y = offset + spread * rng.normal(size=(m, d)), offset + spread * rng.normal(size=(n, d))
    assert np.array_equal(_device_cost(cuda, x, y, 1), _cost(x, y, 1))
    for odd in (np.nan, np.inf):
        x[0, 0], y[n // 2, d - 1] = odd, np.nan
        with np.errstate(invalid="ignore"):
            want = _cost(x, y, 1)
        np.testing.assert_array_equal(_device_cost(cuda, x, y, 1), want)


def test_cost_quotients_are_correctly_rounded(cuda):
    """Many quotients by one divisor, of all magnitudes below it: one-dimensional points against the origin."""
    rng = np.random.default_rng(6)
    x = np.sqrt(np.exp2(rng.uniform(-300, 0, (1_000_000, 1))) * rng.uniform(1, 2, (1_000_000, 1)))
    x[:500_000] = rng.uniform(0.5, 1.4, (500_000, 1))
    y = np.zeros((1, 1))
    assert np.array_equal(_device_cost(cuda, x, y, 1), _cost(x, y))


@pytest.mark.parametrize("m,n,shift", [(1, 1, 0), (2, 300, 0), (255, 31, 0), (256, 33, 0), (514, 65, 1), (513, 129, 0),
                                       (4098, 7, 0), (6, 5000, 0)])
def test_rounding_on_device_buffers(cuda, m, n, shift):
    import torch

    rng = np.random.default_rng(m * n)
    prob = instances.uniform_sqeuclid(m, n, seed=m)
    X = np.outer(prob.source_distribution, prob.target_distribution) * rng.uniform(0, 2, (m, n)) * (rng.random((m, n)) < 0.5)
    X[m // 2] = 0.0  # an empty row: its ratio is a / 0
    lib = _abi.load()
    a, b = (torch.from_numpy(v).to(cuda) for v in (prob.source_distribution, prob.target_distribution))
    buf = torch.zeros(m * n + shift, dtype=torch.float64, device=cuda)
    buf[shift:] = torch.from_numpy(np.ascontiguousarray(X.T)).to(cuda).view(-1)
    _abi.check(lib, lib.pdot_rounding_f64(m, n, a.data_ptr(), b.data_ptr(), buf.data_ptr() + 8 * shift, None), "pdot_rounding_f64")
    torch.cuda.synchronize()
    ref = np.asfortranarray(X)
    oracle.rounding(prob, ref)
    np.testing.assert_allclose(buf[shift:].cpu().numpy().reshape(n, m).T, ref, rtol=1e-12, atol=1e-18)


def _sq(p, q):
    out = np.zeros((p.shape[0], q.shape[0]))
    for k in range(p.shape[1]):
        out += (p[:, k : k + 1] - q[None, :, k]) ** 2
    return out


@pytest.mark.parametrize("offset,spread", [(0.0, 1.0), (1e4, 1e-3), (0.0, 1e-25), (0.0, 1e25)])
@pytest.mark.parametrize("m,n,d", [(1, 1, 1), (513, 1, 2), (700, 257, 3), (1, 4100, 2), (1025, 2049, 1), (256, 64, 2), (129, 2063, 3)])
def test_pair_passes_are_exact(cuda, m, n, d, offset, spread):
    """Bit for bit, also where FP32 tells no pairs apart (an offset, far above the spread) and where its
    squares underflow or overflow."""
    rng = np.random.default_rng(m + 7 * n + d)
    x, y = ((offset + spread * rng.normal(size=(k, d))).astype(np.float32) for k in (m, n))
    x64, y64 = x.astype(np.float64), y.astype(np.float64)
    assert multiscale.max_sq_distance(x, y) == _sq(x64, y64).max()
    centres = offset + spread * rng.normal(size=(n, d))
    dual = spread**2 * rng.normal(size=n)
    got = multiscale.c_transform(x, centres, dual, 0.7)
    assert np.array_equal(got, (0.7 * _sq(x64, centres) - dual[None, :]).min(axis=1))


def test_pair_passes_ignore_what_is_not_a_number(cuda):
    rng = np.random.default_rng(9)
    x, y = rng.normal(size=(600, 2)).astype(np.float32), rng.normal(size=(500, 2)).astype(np.float32)
    centres, dual = rng.normal(size=(500, 2)), rng.normal(size=500)
    y[3, 0], centres[7, 1], dual[9] = np.nan, np.nan, np.nan
    dual[11], dual[12], x[5] = -np.inf, 1e300, np.nan
    with np.errstate(invalid="ignore"):
        far = np.fmax.reduce(_sq(x.astype(np.float64), y.astype(np.float64)), axis=None)
        near = np.fmin.reduce(0.7 * _sq(x.astype(np.float64), centres) - dual[None, :], axis=1, initial=np.inf)
    assert multiscale.max_sq_distance(x, y) == far
    np.testing.assert_array_equal(multiscale.c_transform(x, centres, dual, 0.7), near)


@pytest.mark.parametrize("precision,cost", [("f64", None), ("f32", "f32"), ("f32", "bf16"), ("f32", "sqeuclid"), ("f32", "l1")])
@pytest.mark.parametrize("m,n", [(4739, 33), (35, 4737), (4735, 31), (2367, 29), (2369, 30)])
def test_recovered_plan_of_grouped_rows(cuda, m, n, precision, cost):
    """From 2368 rows (columns) on, 4736 for a stored FP32 or BF16 cost, a warp balances two (four) of
    them; below, one. The balancing's FP32
    exponentials and sums err by some 1e-6 a round and the costs by 2^-9 max C (BF16) or 1e-7, over eps."""
    import pdot

    rng = np.random.default_rng(m)
    xs, ys = rng.uniform(0, 1, (m, 2)).astype(np.float32), rng.uniform(0, 1, (n, 2)).astype(np.float32)
    l1 = cost == "l1"
    C = instances.l1_cost(xs.astype(np.float64), ys.astype(np.float64)) if l1 else instances.sqeuclid_cost(xs, ys)
    if cost == "bf16":  # entries that BF16 holds
        C = np.asfortranarray(np.round(C * 128) / 128)
    a, b = rng.dirichlet(np.ones(m)), rng.dirichlet(np.ones(n))
    u0, v0, eps, rounds = 0.1 * rng.random(m), 0.1 * rng.random(n), 2e-2, 3
    want, _, _ = oracle.warm_plan(C, a, b, u0, v0, eps, rounds)
    kw = {"points": (xs, ys)} if cost in ("sqeuclid", "l1") else {}
    out = pdot.optimize(pdot.default_parameters(1e-4, iteration_limit=0), pdot.OptimalTransportProblem(C, a, b),
                        precision=precision, cost=cost, warm_start=(u0, v0), recover_plan=(eps, rounds), **kw)
    np.testing.assert_allclose(out.primal_solution, want, rtol=1e-3, atol=1e-12)


def test_recovered_plans_of_a_batch_whose_groups_cross_instances(cuda):
    import pdot

    probs, pts = instances.batched_l1(80, 41, 95, seed=3)
    rng = np.random.default_rng(1)
    warm = [(0.1 * rng.random(p.source_distribution.size), 0.1 * rng.random(p.target_distribution.size)) for p in probs]
    warm[1] = warm[40] = None  # cold instances in between
    eps, rounds = 2e-2, 3
    outs, _ = pdot.optimize_batched(pdot.default_parameters(1e-4, iteration_limit=0), probs, cost="l1", points=pts,
                                    warm_starts=warm, recover_plan=(eps, rounds))
    for p, (x, y), w, o in zip(probs, pts, warm, outs):
        if w is None:
            assert not o.primal_solution.any()
            continue
        C = instances.l1_cost(x.astype(np.float32).astype(np.float64), y.astype(np.float32).astype(np.float64))
        want, _, _ = oracle.warm_plan(C, p.source_distribution, p.target_distribution, w[0], w[1], eps, rounds)
        np.testing.assert_allclose(o.primal_solution, want, rtol=1e-3, atol=1e-12)


@pytest.mark.parametrize("dims,batch", [((128, 128, 128), 1), ((2048, 128, 128), 130), ((1024, 256, 384), 257),
                                        ((4096, 128, 256), 128), ((256, 1024, 512), 513)])
def test_network_step_at_odd_shapes(cuda, dims, batch):
    """A training step against the network's oracle for products split 1 to 16 ways over a cluster and for
    batches that end inside a tile: outputs to 1e-3 and gradients to 1e-2 in the 2-norm, as at full size,
    and the loss, summed in FP64 over FP32 differences, to 1e-4."""
    import mlp_oracle as mo
    import torch

    from pdot import learned

    I, H, O = dims
    rng = np.random.default_rng(I + batch)
    net = learned.MLP(I, H, O, max_batch=batch, seed=3)
    hist = np.exp(rng.normal(size=(batch, I)))
    hist /= hist.sum(1, keepdims=True)
    target = rng.normal(size=(batch, O)).astype(np.float32)
    h, t = torch.from_numpy(hist).to(cuda), torch.from_numpy(target).to(cuda)
    y = torch.zeros((batch, O), dtype=torch.float32, device=cuda)
    theta = net.get_parameters()
    torch.cuda.synchronize()
    net.set_input(h.data_ptr(), batch)
    net.forward(y.data_ptr())
    loss = net.backward(t.data_ptr())
    x = mo.features(hist, learned.FEATURE_SHIFT, learned.FEATURE_SCALE)
    want_y, _ = mo.forward(theta, x, I, H, O)
    want_loss, want_g = mo.loss_and_gradients(theta, x, target, I, H, O)
    assert np.linalg.norm(y.cpu().numpy() - want_y) <= 1e-3 * np.linalg.norm(want_y)
    assert loss == pytest.approx(want_loss, rel=1e-4)
    g = net.gradients()
    sizes = [H * I, H, H * H, H, O * H, O]
    for name, lo, k in zip(["W1", "b1", "W2", "b2", "W3", "b3"], np.cumsum([0] + sizes), sizes):
        assert np.linalg.norm(g[lo : lo + k] - want_g[lo : lo + k]) <= 1e-2 * np.linalg.norm(want_g[lo : lo + k]), name


@pytest.mark.parametrize("m,n", [(256, 47359), (256, 47360), (256, 94720), (257, 47360), (255, 94721), (2048, 36000)])
def test_primal_pass_where_its_grid_grows(cuda, m, n):
    """The stand-alone pass around the sizes at which its grid becomes a multiple of the resident CTAs (160
    units a CTA range, two ranges per SM): entries bit for bit, sums to 1e-12 of their terms' magnitude."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(m + n)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    C, X, Xa, u, v = rand(n, m), rand(n, m), rand(n, m), rand(m), rand(n)
    dr, dc, dq = torch.empty(m, dtype=torch.float64, device=cuda), torch.empty(n, dtype=torch.float64, device=cuda), torch.empty(1, dtype=torch.float64, device=cuda)
    s, nw, aw = 0.3, 0.25, 0.8
    D = (X - s * ((C - u[None, :]) - v[:, None])).clamp(min=0.0) - X
    want_x = X + D
    want_a = (Xa + want_x * nw) * aw
    lib = _abi.load()
    need = lib.pdot_primal_pass_workspace_bytes(m, n)
    work = torch.empty(need, dtype=torch.uint8, device=cuda)
    torch.cuda.synchronize()
    _abi.check(lib, lib.pdot_primal_pass_f64(m, n, C.data_ptr(), X.data_ptr(), Xa.data_ptr(), u.data_ptr(), v.data_ptr(), s, nw,
                                             aw, 0, dr.data_ptr(), dc.data_ptr(), dq.data_ptr(), work.data_ptr(), need, None),
               "pdot_primal_pass_f64")
    torch.cuda.synchronize()
    assert torch.equal(X, want_x) and torch.equal(Xa, want_a)
    assert (dr - D.sum(0)).abs().max() <= 1e-12 * D.abs().sum(0).max()
    assert (dc - D.sum(1)).abs().max() <= 1e-12 * D.abs().sum(1).max()
    assert abs(float(dq - D.square().sum())) <= 1e-12 * float(D.square().sum())
