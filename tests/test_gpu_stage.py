"""RK4 and Euler stages of the tiled kernel against the right-hand side of
single cells (rk4_step, src/solver/advancer.py:41-113), bit for bit: rows of
aligned 16-byte chunks and others, partial tiles, short marches."""
import pytest
import torch

from pyflow_b200 import ops

pytestmark = pytest.mark.gpu

SP, MU, RHO, DT = (0.05, 0.07, 0.06), 0.005, 1.3, 0.003


def _field(shape, seed, shift):
    g = torch.Generator("cuda").manual_seed(seed)
    n = shape[0] * shape[1] * shape[2]
    flat = torch.empty(n + shift, dtype=torch.float64, device="cuda")
    out = flat[shift:].view(shape)
    out.copy_(torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 0.5)
    return out


def _steps(f, dtype, rk4):
    """The step by rhs_ns of whole fields in the stage type."""
    def rhs(s):
        return ops.rhs_ns(*[t.to(dtype).clone() for t in s], SP, MU, RHO)
    k = rhs(f)
    if not rk4:
        return [u + q.double() * DT for u, q in zip(f, k)]
    h, acc = 0.5 * DT, list(k)
    for _ in range(2):
        s = [(h * q.double() + u).to(dtype) for u, q in zip(f, k)]
        k = rhs(s)
        acc = [a + 2.0 * q for a, q in zip(acc, k)]
    s = [(h * q.double() + u).to(dtype) for u, q in zip(f, k)]
    # the stage-4 state is u + dt/2 k3
    k = rhs(s)
    return [u + (DT / 6.0) * (a + q).double() for u, a, q in zip(f, acc, k)]


@pytest.mark.parametrize("rk4", [True, False])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("shape,shift", [
    ((3, 3, 4), 0), ((5, 17, 32), 0), ((5, 17, 32), 1), ((7, 16, 36), 0), ((4, 33, 31), 0),
    ((6, 15, 34), 0), ((6, 15, 34), 1), ((130, 9, 28), 0), ((40, 64, 100), 0)])
def test_stage_bits(shape, shift, prec, rk4):
    f = [_field(shape, 7 + q, shift) for q in range(3)]
    ref = _steps(f, torch.float64 if prec == "fp64" else torch.float32, rk4)
    ops.predictor_step(*f, SP, MU, RHO, DT, rk4=rk4, prec=prec)
    for a, b in zip(f, ref):
        assert torch.equal(a, b)
