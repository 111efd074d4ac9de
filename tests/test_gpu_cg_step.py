"""The two-kernel PCG of the levels above the resident solve's limit: after n
iterations its x against the same iterations in 64 bits, for n on every slot of
the ring of search directions and past its end, with and without neighbour
terms, on extents that no tile divides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cg64(i0, i1, smooth, energy, n):
    """n iterations of the Jacobi-PCG of optflow4d.cpp:268-329 in FP64."""
    import torch

    X = i0.shape[3]
    a, b = (torch.from_numpy(v).cuda().double() for v in (i0, i1))
    inner = (slice(1, -1),) * 4
    g = torch.zeros(b.shape + (4,), device="cuda", dtype=torch.float64)
    for c, ax in enumerate((3, 2, 1, 0)):
        g[inner + (c,)] = ((torch.roll(b, -1, ax) - torch.roll(b, 1, ax)) * (X / 2.0))[inner]
    diag = 8 * smooth + energy
    r, pre, x = torch.zeros_like(g), torch.zeros_like(g), torch.zeros_like(g)
    r[inner] = (-g * (b - a).unsqueeze(-1))[inner]
    pre[inner] = (1.0 / (g * g + diag))[inner]
    p = pre * r
    sigma = (p * r).sum()
    for _ in range(n):
        q = torch.zeros_like(p)
        nb = sum(torch.roll(p, k, ax) for ax in range(4) for k in (-1, 1))
        q[inner] = (g * (g * p).sum(-1, keepdim=True) + diag * p - smooth * nb)[inner]
        alpha = sigma / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        z = pre * r
        new = (z * r).sum()
        p = z + (new / sigma) * p
        sigma = new
    return (x * X).cpu().numpy()


@pytest.mark.parametrize("dims", [(134, 133, 132, 3), (43, 45, 41, 42)])
@pytest.mark.parametrize("smooth", [0.001, 0.0])
def test_steps_match_64_bits(dims, smooth):
    import ofblend_gb300 as F

    X, Y, Z, T = dims
    rng = np.random.default_rng(sum(dims))
    base = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
    for ax in range(4):  # a smooth field of the solver's input magnitude
        base = (base + np.roll(base, 1, ax)).astype(np.float32) * np.float32(0.5)
    i0 = base * np.float32(0.02)
    i1 = np.roll(i0, 1, axis=3) + np.float32(0.001)
    g0, g1 = F.Grid4Real(dims=dims).from_numpy(i0), F.Grid4Real(dims=dims).from_numpy(i1)
    v = F.Grid4Vec4(dims=dims)
    for n in (1, 2, 3, 4, 5, 9):
        v.clear()  # the solve takes its right-hand side from it too
        it, _ = F.opticalFlow4d(v, g0, g1, wSmooth=smooth, wEnergy=0.0001, cgAccuracy=1e-12, cgMaxIter=n)
        assert it == n
        want = cg64(i0, i1, smooth, 0.0001, n)
        got = v.to_numpy().astype(np.float64)
        # q, r, p and x are each rounded at some 20 places an iteration, and an
        # iteration carries the errors of those before it: 3 x 20 x n roundings
        assert np.linalg.norm(got - want) <= 60 * n * 2.0 ** -24 * np.linalg.norm(want)


def test_one_direction_buffer_when_memory_is_short():
    """Where the ring's extra buffers do not fit, the solve keeps one direction
    and adds it to x in every step."""
    import torch

    import ofblend_gb300 as F

    dims = (43, 45, 41, 42)
    X, Y, Z, T = dims
    grid = X * Y * Z * T * 16
    rng = np.random.default_rng(7)
    i0 = (rng.standard_normal((T, Z, Y, X)) * 0.01).astype(np.float32)
    i1 = np.roll(i0, 1, axis=3) + np.float32(0.001)
    want = cg64(i0, i1, 0.001, 0.0001, 5)
    torch.cuda.empty_cache()
    launches = []
    for short in (False, True):
        ctx = F.Context(0)
        g0, g1 = (F.Grid4Real(dims=dims, ctx=ctx).from_numpy(v) for v in (i0, i1))
        v = F.Grid4Vec4(dims=dims, ctx=ctx)
        v.clear()
        ctx.synchronize()
        free = torch.cuda.mem_get_info()[0]
        # g, r, p, q and x fit, and one or two of the three extra buffers
        fill = torch.empty(max(0, free - 7 * grid) if short else 1, dtype=torch.uint8, device="cuda")
        n0 = ctx.kernel_launches()
        F.opticalFlow4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-12, cgMaxIter=5)
        launches.append(ctx.kernel_launches() - n0)
        del fill
        torch.cuda.empty_cache()
        got = v.to_numpy().astype(np.float64)
        assert np.linalg.norm(got - want) <= 60 * 5 * 2.0 ** -24 * np.linalg.norm(want)
    assert launches[1] == launches[0] - 1  # five steps leave one direction in the ring to add, none here
