"""The FP64 BiCGStab in one cooperative launch (up to 296 tiles of at most six
planes) against the launch pairs, which per-kernel timing selects: bitwise the
same DP, iterations, residual and status."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# tile edges in y (16) and z (32) and remainders of one cell, one tile along an
# axis (its own neighbour), partial last x chunks, one and two blocks per SM,
# tiles of 4, 5 and 6 planes
SHAPES = [(2, 2, 2), (3, 5, 4), (4, 16, 32), (5, 17, 33), (9, 16, 31), (8, 15, 64), (21, 33, 20),
          (64, 64, 64), (65, 48, 64), (70, 90, 50), (100, 88, 36), (96, 96, 96), (61, 100, 96)]


def _solve(src, sp, max_it):
    import pyflow_b200.ops as ops
    DP = torch.full_like(src, 3.0)
    p = torch.ones_like(src)
    info = ops.bicgstab_solve(src, DP, p, sp, 1.0, 0.01, 1e-10, max_it)
    return DP, p, (info.iterations, info.max_res, info.status)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("max_it", [5000, 3])
def test_one_launch_is_the_launch_pairs(shape, max_it):
    import pyflow_b200.ops as ops
    import pyflow_b200.profiling as prof
    rng = np.random.default_rng(sum(shape))
    sp = (0.31, 0.17, 0.23)
    vel = [torch.tensor(rng.standard_normal(shape), device="cuda") for _ in range(3)]
    src = ops.div_vel(*vel, sp)
    one = _solve(src, sp, max_it)
    prof.enable(True)
    pairs = _solve(src, sp, max_it)
    kt = prof.read()
    prof.enable(False)
    assert kt["bicg_b_f64"]["launches"] > 0
    assert torch.equal(one[0], pairs[0]) and torch.equal(one[1], pairs[1])
    assert one[2] == pairs[2]


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_one_launch_stops_on_non_finite(bad):
    src = torch.randn((24, 20, 36), dtype=torch.float64, device="cuda")
    src[1, 2, 3] = bad
    _, _, (its, res, status) = _solve(src, (0.1,) * 3, 500)
    assert status == 5 and its <= 2


def test_one_launch_zero_source():
    src = torch.zeros((24, 20, 36), dtype=torch.float64, device="cuda")
    DP, _, (its, _, status) = _solve(src, (0.1,) * 3, 500)
    assert its == 0 and status == 3 and float(DP.abs().max()) == 0.0
