"""The direct pressure solve by fast transforms (mixed forms; PF_FP64 with
PF_DIRECT_SOLVE): against numpy's FFT of the same operator in FP64 over
extents of every radix, primes, odd pairs and both ends of the range; its
check; and the iterations behind it."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# powers of two (every last radix), 3, 5, 7 and other primes, odd extents in
# each position (unpaired and unaligned lines), two-cell axes, long lines
SHAPES = [(2, 2, 2), (3, 2, 5), (8, 4, 2), (16, 32, 64), (64, 16, 32), (12, 20, 28), (9, 25, 49),
          (15, 7, 33), (21, 34, 11), (13, 17, 19), (31, 6, 10), (10, 37, 5), (6, 10, 61),
          (128, 4, 6), (4, 256, 6), (4, 6, 512), (1024, 3, 4), (2, 1024, 6), (4, 2, 2048),
          (2048, 2, 3), (3, 2048, 2), (96, 80, 72), (4, 1331, 3), (2, 3, 1021), (2039, 2, 2)]


def _solve(src, sp, prec, tol=1e-10, max_it=20000, rho=1.3, dt=0.01, flags=0):
    import pyflow_b200._lib as L
    import pyflow_b200.ops as ops
    DP = torch.full_like(src, 7.0)
    p = torch.ones_like(src)
    g = ops.grid(src.shape, sp)
    pr = ops.PREC[prec]
    ws = ops.workspace(g, pr, src.device)
    info = L.SolveInfo()
    L.check("pf_bicgstab_solve", L.lib().pf_bicgstab_solve(
        ctypes.byref(g), pr | flags, rho, dt, tol, max_it, ops._p(src), ops._p(DP), ops._p(p),
        ops._p(ws), ws.numel(), ops._stream(src), ctypes.byref(info)))
    return DP, p, info


def _exact(src, sp, rho=1.3, dt=0.01):
    """Zero-mean solution of the 7-point Laplacian by numpy's FFT."""
    lam = 0.0
    for d, n in enumerate(src.shape):
        s = [1, 1, 1]
        s[d] = n
        lam = lam - (4.0 / sp[d] ** 2 * np.sin(np.pi * np.arange(n) / n) ** 2).reshape(s)
    lam[0, 0, 0] = 1.0
    h = np.fft.fftn(src) / lam
    h[0, 0, 0] = 0.0
    return np.fft.ifftn(h).real * (rho / dt)


@pytest.mark.parametrize("shape", SHAPES)
def test_direct_solve_matches_fft(shape):
    """FP64 transforms leave a few roundings (2e-16) per stage relative to the
    norm, direct sums of a prime p up to p: 1e-12 of the norm bounds both."""
    rng = np.random.default_rng(sum(shape))
    sp = (0.31, 0.17, 0.23)
    src = rng.standard_normal(shape)
    src -= src.mean()
    want = _exact(src, sp)
    forms = [("mixed", 0), ("fp64", 0x200)]
    if np.prod(shape) > 2 ** 15:
        forms.append(("mixed_mg", 0))   # smaller grids that coarsen keep the V-cycles
    for prec, flags in forms:
        DP, p, info = _solve(torch.tensor(src, device="cuda"), sp, prec, flags=flags)
        assert info.status == 0 and info.iterations == 1 and info.max_res <= 1e-10
        got = DP.cpu().numpy()
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
        assert torch.equal(p, 1.0 + DP)


def test_source_with_a_mean_goes_on_iterating():
    """A right-hand side with a mean has no solution: the direct result
    misses the tolerance, the FP64 passes run to the limit and say so."""
    src = torch.ones(16, 12, 20, dtype=torch.float64, device="cuda")
    src[3, 4, 5] = 2.0
    for prec, flags in (("mixed", 0), ("mixed_mg", 0), ("fp64", 0x200)):
        _, _, info = _solve(src, (0.1,) * 3, prec, max_it=40, flags=flags)
        assert info.status != 0 and info.max_res > 1e-10 and info.iterations >= 1


def test_tight_tolerance_iterates():
    """Below the direct solve's own rounding the iterations run as before."""
    rng = np.random.default_rng(3)
    a = rng.standard_normal((24, 24, 24))
    src = torch.tensor(a - a.mean(), device="cuda")
    _, _, info = _solve(src, (0.1,) * 3, "mixed", tol=2e-13)
    assert info.iterations > 1


def test_unaligned_fields():
    """Fields that start 8 bytes off a 16-byte boundary, even extents."""
    import pyflow_b200.ops as ops
    shape, sp = (16, 12, 10), (0.31, 0.17, 0.23)
    n = int(np.prod(shape))
    rng = np.random.default_rng(9)
    a = rng.standard_normal(shape)
    a -= a.mean()
    buf = [torch.zeros(n + 1, dtype=torch.float64, device="cuda") for _ in range(3)]
    src, DP, p = (b[1:].view(shape) for b in buf)
    src.copy_(torch.tensor(a, device="cuda"))
    info = ops.bicgstab_solve(src, DP, p, sp, 1.3, 0.01, 1e-10, 100, prec="mixed")
    want = _exact(a, sp)
    assert info.status == 0
    assert np.linalg.norm(DP.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("shape", [(40, 36, 24), (21, 20, 33)])
def test_plan_takes_the_correction_back(shape):
    """A box flattened in z whose flow does not vary in z: the rounding of
    A x, times the square of the aspect ratio, is above the tolerance, so the
    step graph's check fails after the correction, which is taken back before
    the FP64 passes run and is applied again.  The limit ends them; velocity
    and pressure are those of the host-driven step, which corrects once."""
    import pyflow_b200.ops as ops
    from pyflow_b200.plan import StepPlan
    sp = (0.2, 0.25, 2e-6)
    rng = np.random.default_rng(5)
    k = [2 * np.pi * np.arange(n) / n for n in shape[:2]]
    f0 = [np.broadcast_to((np.sin(k[0] + a)[:, None] * np.cos(k[1] + b)[None, :])[..., None], shape)
          for a, b in rng.uniform(0, 6, (3, 2))]
    f0 = [torch.tensor(np.ascontiguousarray(x), device="cuda") for x in f0]
    out = []
    for plan in (True, False):
        f = [t.clone() for t in f0] + [torch.zeros_like(f0[0]), torch.zeros_like(f0[0])]
        if plan:
            pl = StepPlan(*f, sp, 0.0, 1.0, 1e-7, min_res=1e-10, max_it=12, prec="mixed")
            pl.launch(1)
            torch.cuda.synchronize()
            st = pl.stats()
            pl.close()
            status, res = int(st["status"]), st["max_res"]
            np.testing.assert_allclose(
                [st[n] for n in ("max_u", "max_v", "max_w", "tke", "max_div")],
                ops.stats(*f[:3], sp).cpu().numpy(), rtol=1e-14)
        else:
            info = ops.forward_step(*f, sp, 0.0, 1.0, 1e-7, min_res=1e-10, max_it=12, prec="mixed")
            status, res = info.status, info.max_res
        out.append((f, status, res))
    (a, sa, ra), (b, sb, rb) = out
    assert sa != 0 and sb != 0 and ra > 1e-10 and rb > 1e-10
    for x, y in zip(a[:4], b[:4]):
        assert torch.isfinite(x).all()
        assert float((x - y).abs().max()) <= 1e-6 * float(y.abs().max())


@pytest.mark.parametrize("n", [32, 64, 96, 128, 160, 192, 256, 320, 384, 512, 640, 768, 1024])
@pytest.mark.parametrize("rest", [(3, 5), (2, 17), (18, 4)])
def test_unrolled_extents_match_fft(n, rest):
    """The extents with stages laid out at compile time, in each position, with
    unpaired, unaligned and partial line groups beside them; bounds as above."""
    for axis in range(3):
        shape = rest[:axis] + (n,) + rest[axis:]
        rng = np.random.default_rng(n + axis)
        sp = (0.31, 0.17, 0.23)
        src = rng.standard_normal(shape)
        src -= src.mean()
        want = _exact(src, sp)
        DP, _, info = _solve(torch.tensor(src, device="cuda"), sp, "fp64", flags=0x200)
        assert info.status == 0 and info.iterations == 1 and info.max_res <= 1e-10
        got = DP.cpu().numpy()
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("prec", ["mixed", "mixed_mg", "fp64"])
@pytest.mark.parametrize("shape", [(24, 20, 36), (64, 64, 64)])
def test_source_and_solution_in_one_buffer(prec, shape):
    """DP in the buffer of the source: the solve reads each cell's source
    before it writes that cell and keeps the right-hand side itself, so the
    result is that of separate buffers.  Each residual is at most 1e-10 max|b|,
    so each error at most 1e-10 kappa max|b| sqrt(N) / |b| of the solution, with
    kappa <= 2600 and max|b| sqrt(N) / |b| <= 5.5 here: 3e-6 for the two."""
    import pyflow_b200.ops as ops
    sp = (0.31, 0.17, 0.23)
    a = np.random.default_rng(1).standard_normal(shape)
    src = torch.tensor(a - a.mean(), device="cuda")
    out = []
    for same in (True, False):
        s = src.clone()
        DP = s if same else torch.empty_like(s)
        p = torch.zeros_like(s)
        info = ops.bicgstab_solve(s, DP, p, sp, 1.3, 0.01, 1e-10, 20000, prec=prec)
        assert info.status == 0 and info.max_res <= 1e-10
        assert torch.equal(p, DP)
        out.append(DP - DP.mean())
    assert float((out[0] - out[1]).norm()) <= 3e-6 * float(out[1].norm())


@pytest.mark.parametrize("prec", ["mixed", "mixed_mg"])
def test_sources_beyond_the_transforms_range(prec):
    """Finite sources whose transforms overflow (their values times the square
    root of the cells): the scaled passes solve them.  The error is at most
    1e-10 kappa max|b| sqrt(N) / |b| of the solution (kappa 1440, 5)."""
    shape, sp = (48, 40, 56), (0.31, 0.17, 0.23)
    a = np.random.default_rng(2).standard_normal(shape)
    a -= a.mean()
    want = _exact(a, sp, 1.0, 1.0)
    DP, p, info = _solve(torch.tensor(a * 1e307, device="cuda"), sp, prec, rho=1.0, dt=1.0)
    assert info.status == 0 and info.max_res <= 1e-10
    got = DP.cpu().numpy() / 1e307
    got -= got.mean()
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    assert torch.equal(p, 1.0 + DP)


def test_right_hand_side_that_overflows():
    """A finite source times an infinite rho/dt: reported, p untouched."""
    a = np.random.default_rng(2).standard_normal((24, 20, 28))
    src = torch.tensor(a - a.mean(), device="cuda")
    DP, p, info = _solve(src, (0.31, 0.17, 0.23), "mixed", rho=1e200, dt=1e-200)
    assert info.status == 5
    assert float(DP.abs().max()) == 0.0 and torch.equal(p, torch.ones_like(p))


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("prec,flags", [("mixed", 0), ("mixed_mg", 0), ("fp64", 0x200)])
def test_non_finite_source(value, prec, flags):
    """One non-finite cell: reported, DP = 0 and p untouched."""
    src = torch.randn(48, 40, 56, dtype=torch.float64, device="cuda")
    src[3, 7, 11] = value
    DP, p, info = _solve(src, (0.31, 0.17, 0.23), prec, flags=flags)
    assert info.status == 5
    assert float(DP.abs().max()) == 0.0 and torch.equal(p, torch.ones_like(p))


def test_tight_tolerance_is_reached():
    """Below the direct solve's tolerance the iterations reach theirs: the true
    residual (evaluated again: a few roundings of the operator's largest
    terms, kappa times |b|), and with it the solution: |error| <= |r| / least
    eigenvalue in the 2-norm, |r| <= sqrt(N) max|r|."""
    import pyflow_b200.ops as ops
    n, h, tol, c1 = 24, 0.1, 2e-13, 1.3 / 0.01
    a = np.random.default_rng(3).standard_normal((n,) * 3)
    a -= a.mean()
    src, sp = torch.tensor(a, device="cuda"), (h,) * 3
    DP, _, info = _solve(src, sp, "mixed", tol=tol)
    assert info.status == 0 and info.iterations > 1
    s2 = np.sin(np.pi / n) ** 2
    b = src * c1 * -(h ** 3)
    res = float((b - ops.laplace_apply(DP, sp)).abs().max() / b.abs().max())
    assert res <= tol + 8 * 2.0 ** -53 * 3 / s2
    got, want = DP.cpu().numpy(), _exact(a, sp)
    got -= got.mean()
    bound = tol * np.sqrt(a.size) * np.abs(a).max() * c1 * h ** 2 / (4 * s2)
    assert np.linalg.norm(got - want) <= bound + 1e-15 * np.linalg.norm(want)


@pytest.mark.parametrize("shape", [(40, 36, 24), (21, 20, 33)])
def test_correction_taken_back_costs_its_roundings(shape):
    """The flattened box of test_plan_takes_the_correction_back, first step:
    the graph's velocity went through the rejected correction c0 = dt/rho grad
    DP0 and back, the host-driven one did not, and both then take the same
    correction.  Each of the two extra operations rounds a value of at most
    |u| + 2 |c0| once, and differing inputs of the last one can round apart
    once more: 4 units of 2^-53 of |u| + 2 |c0| + |c1| (c1: the final
    correction), beside what the two DP themselves differ by; the pressure
    likewise with DP0 and DP1."""
    import pyflow_b200.ops as ops
    from pyflow_b200.plan import StepPlan
    sp, dt = (0.2, 0.25, 2e-6), 1e-7
    rng = np.random.default_rng(5)
    k = [2 * np.pi * np.arange(n) / n for n in shape[:2]]
    f0 = [np.broadcast_to((np.sin(k[0] + a)[:, None] * np.cos(k[1] + b)[None, :])[..., None], shape)
          for a, b in rng.uniform(0, 6, (3, 2))]
    f0 = [torch.tensor(np.ascontiguousarray(x), device="cuda") for x in f0]
    z = lambda: torch.zeros_like(f0[0])  # noqa: E731
    a, b = [t.clone() for t in f0] + [z(), z()], [t.clone() for t in f0] + [z(), z()]
    info = ops.forward_step(*a, sp, 0.0, 1.0, dt, min_res=1e-10, max_it=12, prec="mixed")
    plan = StepPlan(*b, sp, 0.0, 1.0, dt, min_res=1e-10, max_it=12, prec="mixed")
    plan.launch(1)
    torch.cuda.synchronize()
    assert plan.stats()["status"] != 0 and info.status != 0
    plan.close()
    # the rejected correction: the direct solve of the same divergence alone
    c = [t.clone() for t in f0]
    ops.predictor_step(*c, sp, 0.0, 1.0, dt, prec="mixed")
    DP0, p = z(), z()
    ops.bicgstab_solve(ops.div_vel(*c, sp), DP0, p, sp, 1.0, dt, 1e-10, 1, prec="mixed")

    def grad(f, d):
        return dt * (f - f.roll(1, d)) / sp[d]
    for d in range(3):
        bound = 4 * 2.0 ** -53 * (c[d].abs() + 2 * grad(DP0, d).abs() + grad(a[4], d).abs())
        bound += grad(a[4] - b[4], d).abs()
        assert bool(((a[d] - b[d]).abs() <= bound).all())
    bound = 4 * 2.0 ** -53 * (2 * DP0.abs() + a[4].abs()) + (a[4] - b[4]).abs()
    assert bool(((a[3] - b[3]).abs() <= bound).all())
