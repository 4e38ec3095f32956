"""Products, bias sums and Adam steps of several layers in one launch against
the same ones launched by themselves, word for word, and the tiled elementwise
kernels at sizes that are no multiple of their 32 x 32 tiles."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.float32):
    return torch.randn(*shape, device="cuda", generator=_rand.gen).to(dtype)


@pytest.fixture(autouse=True)
def _seed():
    assert torch.cuda.is_available()
    _rand.gen = torch.Generator(device="cuda").manual_seed(5)


# one product; as many as a launch takes; one more
@pytest.mark.parametrize("n", [1, 8, 9])
@pytest.mark.parametrize("bn", [128, 256])
def test_grouped_products_equal_single_ones(n, bn):
    from hexdyn import mlp

    sizes = [((128, 64), (256, 64)), ((384, 192), (512, 192)), ((256, 1024), (256, 1024))]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    problems, singles, groups = [], [], []
    for i in range(n):
        a, b = (_rand(*s, dtype=torch.bfloat16) for s in sizes[i % 3])
        one, many = (torch.full((a.shape[0], b.shape[0]), float("nan"), device="cuda") for _ in range(2))
        mlp.gemm(a, b, epilogue=mlp.EPI_F32, Cf=one, err=err, bn=bn)
        problems.append(mlp._problem(a, b, bn, mlp.EPI_F32, None, None, None, None, None, many, err,
                                     mlp.GEMM_PERSISTENT))
        singles.append((one, a, b))
        groups.append(many)
    assert mlp.load().hexmlp_gemm_group((mlp.HexMlpGemm * n)(*problems), n, mlp._stream()) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    for (one, a, b), many in zip(singles, groups):
        assert torch.equal(one, many)
        # 2^-24 per step of a 32-bit sum of K products, with room for the order
        bound = 2.0 ** -24 * a.shape[1] * (a.double().abs() @ b.double().abs().t())
        assert bool(((many.double() - a.double() @ b.double().t()).abs() <= bound).all())


def test_a_group_with_a_refused_product_launches_nothing():
    from hexdyn import mlp

    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = _rand(128, 64, dtype=torch.bfloat16)
    out = torch.zeros(128, 128, device="cuda")
    good = mlp._problem(a, a, 128, mlp.EPI_F32, None, None, None, None, None, out, err, mlp.GEMM_PERSISTENT)
    for change in (dict(M=100), dict(kernel=mlp.GEMM_STAGED), dict(Cf=None), dict(bn=256)):
        bad = mlp.HexMlpGemm.from_buffer_copy(good)
        for k, v in change.items():
            setattr(bad, k, v)
        assert mlp.load().hexmlp_gemm_group((mlp.HexMlpGemm * 2)(good, bad), 2, mlp._stream()) == -1
    torch.cuda.synchronize()
    assert not bool(out.any())


@pytest.mark.parametrize("M, N", [(1, 1), (31, 33), (96, 65), (128, 256)])
def test_loss_gradient_tiles(M, N):
    from hexdyn import mlp

    Y, T = _rand(M, N), _rand(M, N)
    dY = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    dYt = torch.zeros(N, M, dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(1, device="cuda")
    mv, nv = max(1, M - 3), max(1, N - 2)
    p = mlp._ptr
    assert mlp.load().hexmlp_mse_grad(p(Y), p(T), M, N, mv, nv, 0.25, p(dY), p(dYt), p(loss), mlp._stream()) == 0
    want = torch.zeros(M, N, device="cuda")
    want[:mv, :nv] = 2.0 * (Y - T)[:mv, :nv] * 0.25
    assert torch.equal(dY, want.to(torch.bfloat16)) and torch.equal(dYt, dY.t())
    exact = float((Y - T)[:mv, :nv].double().square().sum())
    assert abs(float(loss) - exact) <= 2.0 ** -23 * (mv * nv) ** 0.5 * 8 * max(exact, 1e-30)


# more arrays than a launch's sixteen, among them a bias and odd sizes
@pytest.mark.parametrize("n", [1, 17])
def test_layers_in_one_launch_equal_single_steps(n):
    from hexdyn import mlp

    lib, p = mlp.load(), mlp._ptr
    shapes = [(33, 31), (1, 70), (128, 64)]
    parts, kept = [], []
    for i in range(n):
        rows, cols = shapes[i % 3]
        w, m1, g = (_rand(rows, cols) for _ in range(3))
        m2 = _rand(rows, cols).square()
        both = [[t.clone() for t in (w, m1, m2)] + [torch.zeros(rows, cols, dtype=torch.bfloat16, device="cuda"),
                                                  torch.zeros(cols, rows, dtype=torch.bfloat16, device="cuda")]
                for _ in range(2)]
        a, b = both
        assert lib.hexmlp_adam(p(a[0]), p(a[1]), p(a[2]), p(g), rows, cols, 1e-3, 0.9, 0.999, 1e-8, 3, 0.01, p(a[3]),
                               p(a[4]), mlp._stream()) == 0
        parts.append(mlp.HexMlpAdam(p(b[0]), p(b[1]), p(b[2]), p(g), p(b[3]), p(b[4]), rows, cols, 0.01))
        kept.append((a, b, g))
    assert lib.hexmlp_adam_layers((mlp.HexMlpAdam * n)(*parts), n, 1e-3, 0.9, 0.999, 1e-8, 3, mlp._stream()) == 0
    torch.cuda.synchronize()
    for a, b, _ in kept:
        assert all(torch.equal(x, y) for x, y in zip(a, b))
        assert torch.equal(b[3], b[0].to(torch.bfloat16)) and torch.equal(b[4], b[3].t())
    dts = [_rand(5 + 3 * i, 200, dtype=torch.bfloat16) for i in range(n)]
    dbs = [torch.zeros(t.shape[0], device="cuda") for t in dts]
    assert lib.hexmlp_bias_grads((C.c_void_p * n)(*map(p, dts)), (C.c_int * n)(*[t.shape[0] for t in dts]),
                                 (C.c_void_p * n)(*map(p, dbs)), n, 200, mlp._stream()) == 0
    for t, db in zip(dts, dbs):
        one = torch.zeros_like(db)
        assert lib.hexmlp_bias_grad(p(t), t.shape[0], 200, p(one), mlp._stream()) == 0
        assert torch.equal(one, db)
        exact = t.double().sum(1)
        bound = 2.0 ** -24 * 200 * t.double().abs().sum(1)
        assert bool(((db.double() - exact).abs() <= bound).all())


def _fma32(a, b, c):
    """a b + c of float32 arrays rounded once: the product is exact in 64 bits,
    and the sum rounded to odd there rounds to float32 as the exact sum does."""
    x, y = a.astype(np.float64) * b.astype(np.float64), np.asarray(c, np.float64)
    s = x + y
    t = s - x
    err = (x - (s - t)) + (y - t)
    even = (s.view(np.int64) & 1) == 0
    s = np.where((err != 0) & even, np.nextafter(s, np.where(err > 0, np.inf, -np.inf)), s)
    return s.astype(np.float32)


# one rounding per operation and the three contractions that the kernel writes out
@pytest.mark.parametrize("decay", [0.0, 0.01, 0.3])
def test_adam_rounds_as_written(decay):
    from hexdyn import mlp

    p, f = mlp._ptr, np.float32
    w, m1, g = (_rand(65, 97) for _ in range(3))
    m2 = _rand(65, 97).square()
    lr, b1, b2, eps = f(1e-3), f(0.9), f(0.999), f(1e-8)
    hw, h1, h2, hg = (t.cpu().numpy() for t in (w, m1, m2, g))
    gi = _fma32(np.full_like(hw, f(decay)), hw, hg)
    m = _fma32(np.full_like(hw, b1), h1, (f(1) - b1) * gi)
    v = _fma32(np.full_like(hw, b2), h2, ((f(1) - b2) * gi) * gi)
    # the first step: the bias corrections are 1 - b1 and 1 - b2
    want = hw - lr * (m / (f(1) - b1)) / (np.sqrt(v / (f(1) - b2)) + eps)
    assert mlp.load().hexmlp_adam(p(w), p(m1), p(m2), p(g), 65, 97, float(lr), float(b1), float(b2), float(eps), 1,
                                  decay, None, None, mlp._stream()) == 0
    for got, expect in ((m1, m), (m2, v), (w, want)):
        assert expect.dtype == np.float32
        assert np.array_equal(got.cpu().numpy().view(np.uint32), expect.view(np.uint32))
