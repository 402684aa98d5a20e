"""The recovery's blocked factorisation at the sizes where its blocks end, and the adjoint's rate-table sum at the batch
sizes where its chunks change."""

import numpy as np
import pytest
import torch

import invented
from maxichem_b200 import coupling
from maxichem_b200.ad import ADSolver
from maxichem_b200.solver import CudaSolver
from test_gpu_lu import isomers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [2, 4])
@pytest.mark.parametrize("species", [3, 8, 9, 17, 33, 41, 64, 65, 97, 130])
def test_recovered_cells_match_the_plain_call(gpu, tmp_path, species, warps):
    net = isomers(tmp_path, species)
    rng = np.random.default_rng(2)
    x = rng.uniform(0.1, 1.0, (24, species))
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=gpu)  # noqa: E731
    args = [t(x / x.sum(1, keepdims=True)), t(rng.uniform(500.0, 1500.0, 24)), t(np.full(24, 1e4)),
            t(np.full(24, 1e-3)), t(np.full(24, 1e-7))]  # fmt: skip
    with CudaSolver(net, gpu, warps=warps) as plain, CudaSolver(net, gpu, warps=warps, drift=0.0) as strict:
        a = plain.launch(*args)
        b = strict.launch(*args)  # no drift allowed: rounding alone sends most cells through the recovery
    assert bool(a.done.all()) and int((b.flag > 0).sum()) > 0
    again = (b.flag > 0).cpu().numpy()
    xa, xb = a.x.cpu().numpy()[again], b.x.cpu().numpy()[again]
    # the same steps with another factorisation of the same matrices: rounding times the stiffness, as between orders
    # of summation elsewhere (1e-9); the guard's correction of the plain result is of the size of its rounding
    assert np.abs(xa - xb).max() <= 1e-9 and np.array_equal(a.steps.cpu().numpy()[again], b.steps.cpu().numpy()[again])


@pytest.mark.parametrize("cells", [1, 7, 1000, 4001])
def test_the_rate_tables_cotangent_is_the_sum_over_the_cells(gpu, tmp_path, cells):
    net, _ = invented.hydrogen(tmp_path)
    rng = np.random.default_rng(cells)
    x = rng.uniform(0.1, 1.0, (cells, len(net.species)))
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=gpu)  # noqa: E731
    args = [t(x / x.sum(1, keepdims=True)), t(rng.uniform(800.0, 1500.0, cells)), t(np.full(cells, 1e5)),
            t(np.full(cells, 1e-6)), t(np.full(cells, 1e-9))]  # fmt: skip
    gx = t(rng.standard_normal(x.shape))
    with ADSolver(net, gpu) as solver:
        whole = solver.vjp(*args, gx).cotangents.rc
        assert bool((solver.flag == 0).all())
        cuts = [0, cells // 3, cells // 2, cells]
        parts = [solver.vjp(*(a[i:j].clone() for a in args), gx[i:j].clone()).cotangents.rc
                 for i, j in zip(cuts, cuts[1:]) if j > i]  # fmt: skip
    total = torch.stack(parts).sum(0)
    # another order of the same terms: at most a rounding per cell of the largest partial sum
    scale = torch.stack(parts).abs().amax(0).clamp_min(1e-300)
    assert float(((whole - total).abs() / scale).max()) <= cells * 4 * 2.3e-16 * 10


@pytest.mark.parametrize("cells", [1, 9, 9473])
@pytest.mark.parametrize("species", [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225, 254])
def test_conversions_at_the_sizes_where_a_lanes_rows_change(gpu, species, cells):
    rng = np.random.default_rng(species + cells)
    q, mw = 10.0 ** rng.uniform(-12.0, 0.0, (cells, species)), rng.uniform(1e-3, 1e-1, species)
    mass = rng.uniform(0.5, 1.5, cells)
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=gpu)  # noqa: E731
    x = coupling.mass_to_mole(t(q), t(mw))
    back = coupling.mole_to_mass(x, t(mw), t(mass)).cpu().numpy()
    n = q / mw
    ref = n / n.sum(1, keepdims=True)
    xm = ref * mw
    want = xm * (mass / xm.sum(1))[:, None]
    # positive sums of at most 254 terms in two orders (254 x 1.1e-16), a few roundings beside
    for got, exact in ((x.cpu().numpy(), ref), (back, want)):
        assert np.abs(got - exact).max() <= 6e-14 * exact.max() and (np.abs(got / exact - 1.0) <= 6e-14).all()


def chunked(net, gpu, cells: int, **options):
    """A solver, a batch and its cotangents for the tests of the rate table's sum."""
    rng = np.random.default_rng(cells)
    x = rng.uniform(0.1, 1.0, (cells, len(net.species)))
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=gpu)  # noqa: E731
    args = [t(x / x.sum(1, keepdims=True)), t(rng.uniform(800.0, 1500.0, cells)), t(np.full(cells, 1e5)),
            t(np.full(cells, 1e-6)), t(np.full(cells, 1e-9))]  # fmt: skip
    return ADSolver(net, gpu, **options), args, t(rng.standard_normal(x.shape))


# a cell a queue item up to 256 times the resident CTAs (113,664 or 151,552 cells), 64 above
@pytest.mark.parametrize("cells", [64, 65, 1000, 4001, 60000, 200000])
def test_the_rate_tables_cotangent_adds_fixed_chunks_of_64_cells_in_order(gpu, tmp_path, cells):
    net, _ = invented.hydrogen(tmp_path)
    solver, args, gx = chunked(net, gpu, cells)
    chunks = -(-cells // 64)
    used = range(chunks) if chunks <= 70 else [0, 1, chunks // 2, chunks - 2, chunks - 1]
    keep = torch.zeros(cells, 1, dtype=torch.bool, device=gpu)
    for k in used:
        keep[64 * k : 64 * (k + 1)] = True
    gx = torch.where(keep, gx, 0.0)  # the other chunks add zeros
    with solver:
        whole = solver.vjp(*args, gx).cotangents.rc
        assert bool((solver.flag == 0).all()) and float(whole.abs().max()) > 0.0
        total = torch.zeros_like(whole)
        for k in used:
            of = slice(64 * k, min(64 * (k + 1), cells))
            total = total + solver.vjp(*(a[of].clone() for a in args), gx[of].clone()).cotangents.rc
    assert torch.equal(whole, total)


def test_recovered_cells_follow_their_chunk_in_the_rate_tables_sum(gpu, tmp_path):
    net, _ = invented.hydrogen(tmp_path)
    solver, args, gx = chunked(net, gpu, 150, drift=0.0)  # no drift allowed: many cells go through the recovery
    with solver:
        whole = solver.vjp(*args, gx).cotangents.rc[:, 0::3]  # the columns whose terms are the cells' own values
        flag = solver.flag.tolist()
        own = [solver.vjp(*(a[i : i + 1].clone() for a in args), gx[i : i + 1].clone()).cotangents.rc[:, 0::3]
               for i in range(150)]  # fmt: skip
    assert 0 in flag and 1 in flag
    total = torch.zeros_like(whole)
    for start in range(0, 150, 64):
        cells = range(start, min(start + 64, 150))
        passed = [own[i] for i in cells if flag[i] == 0]
        total = total + sum(passed[1:], passed[0]) if passed else total
        for i in cells:
            total = total + own[i] if flag[i] == 1 else total
    assert torch.equal(whole, total)
