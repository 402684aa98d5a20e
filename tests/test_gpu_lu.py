"""The factorisation and the triangular solves of one try at the sizes where their blocks end: 8 x 8 tiles, 4-pivot
blocks, 32 rows a lane. Networks of n isomers exchanging on collisions, each with several partners."""

import numpy as np
import pytest
import torch

import invented
import oracle
from maxichem_b200 import abi
from maxichem_b200.solver import CudaSolver

pytestmark = pytest.mark.gpu


def isomers(folder, species: int):
    """species - 1 isomers and He; isomer i exchanges with i + 1, i + 2 and i + 5, rates over four orders."""
    n, rng, lines = species - 1, np.random.default_rng(species), []
    for i in range(n):
        for step in (1, 2, 5):
            if i + step < n or (step == 1 and n > 1 and i == n - 1 and n > 2):
                j = (i + step) % n
                rate = 10.0 ** rng.uniform(-13.0, -9.0)
                lines.append(f"{2 * len(lines) + 1} [ CO_{i + 1} + He -> CO_{j + 1} + He ] {rate:.4E} 0 0")
    thermo = {f"CO_{i + 1}": invented.constant_cp(rng.uniform(-800.0, 800.0)) for i in range(n)}
    thermo["He"] = invented.constant_cp(0.0, 2.5)
    return invented.write(folder, "# Invented: isomers\n# Two-body Reactions\n" + "\n".join(lines) + "\n", thermo)


@pytest.mark.parametrize("warps", [2, 4])
@pytest.mark.parametrize("species", [3, 7, 8, 9, 12, 16, 17, 31, 32, 33, 36, 41, 64, 65, 70, 91, 97, 130])
def test_factors_and_solves_match_the_oracle(gpu, tmp_path, species, warps):
    net = isomers(tmp_path, species)
    assert len(net.species) == species
    rng = np.random.default_rng(1)
    x = rng.uniform(0.1, 1.0, species)
    x /= x.sum()
    with CudaSolver(net, gpu, warps=warps) as solver:
        out = torch.empty(oracle.debug_size(solver.tab), dtype=torch.float64, device=gpu)
        xg = torch.tensor(x, dtype=torch.float64, device=gpu)
        for h in (1e-9, 1e-5):  # the diagonal leads; the rates lead
            assert abi.library().mx_debug_try(solver._handle, xg.data_ptr(), 900.0, 1e4, h, None, 1e-3, 1e-25,
                                              out.data_ptr(), None) == 0  # fmt: skip
            torch.cuda.synchronize()
            g = oracle.split_debug(solver.tab, out.cpu().numpy())
            r = oracle.Oracle(solver.tab).debug_try(x, 900.0, 1e4, h)
            for k in ("LU", "dinv", "K1", "K2", "K3", "K4"):
                # the two sides' rates differ in the last bits of exp (a few ulp); the solves amplify that by the
                # condition of M0, at most about 2 h max(-Jn) + 1 < 1e4 here. Later stages are differences of terms as
                # large as K1, so all four are judged on K1's scale.
                scale = np.abs(r["K1" if k[0] == "K" else k]).max()
                assert np.abs(g[k] - r[k]).max() <= 1e-10 * scale, (species, warps, h, k)


def factored(solver, gpu, a, y, u, c0: float, pivoted: bool):
    """mx_debug_lu's factors, 1 / pivots, row order, solution and corrected solution."""
    n = len(y)
    out = torch.empty(n * n + 4 * n, dtype=torch.float64, device=gpu)
    ag, yg, ug = (torch.tensor(q, dtype=torch.float64, device=gpu) for q in (a, y, u))
    assert abi.library().mx_debug_lu(solver._handle, ag.data_ptr(), yg.data_ptr(), ug.data_ptr(), c0, int(pivoted),
                                     out.data_ptr(), None) == 0  # fmt: skip
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    return o[: n * n].reshape(n, n), *o[n * n :].reshape(4, n)


SIZES = [3, 7, 8, 9, 12, 16, 17, 31, 32, 33, 36, 41, 64, 65, 70, 91, 97, 128, 130]


@pytest.mark.parametrize("warps", [2, 4])
@pytest.mark.parametrize("species", SIZES)
def test_factors_and_solves_have_the_oracles_bits(gpu, tmp_path, species, warps):
    rng = np.random.default_rng(species)
    a = rng.standard_normal((species, species)) * 10.0 ** rng.uniform(-4.0, 4.0, (species, species))
    a += np.diag(10.0 ** rng.uniform(2.0, 6.0, species))
    y, u = rng.standard_normal((2, species))
    with CudaSolver(isomers(tmp_path, species), gpu, warps=warps) as solver:
        lu, dinv, order, x, w = factored(solver, gpu, a, y, u, 0.37, False)
    ref_lu, ref_dinv = oracle.lu(a)
    ref_x = oracle.lu_solve(ref_lu, ref_dinv, y)
    assert np.isfinite(ref_x).all() and np.array_equal(order, np.arange(species))
    # the same correctly rounded operations in the same order: no tolerance, whatever the matrix's condition
    assert np.array_equal(lu, ref_lu) and np.array_equal(dinv, ref_dinv)
    assert np.array_equal(x, ref_x) and np.array_equal(w, oracle.sherman(ref_x, u, 0.37))


def matrices(n: int):
    """Matrices for the threshold rule: name, matrix."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    yield "exchanges", a
    yield "none", a + 50.0 * n * np.eye(n)
    yield "ties", rng.integers(-1, 2, (n, n)) + 0.0
    late = a.copy()  # its columns' largest entries in the last rows: exchanges over every block
    late[-(-n // 2) :] *= 1e3
    yield "far", late
    zero = a.copy()
    zero[:, n // 2] = 0.0  # no pivot there: infinities and NaN from that column on
    yield "zero column", zero
    nan = a.copy()
    nan[n - 1, n // 2] = np.nan
    yield "nan", nan


@pytest.mark.parametrize("warps", [2, 4])
@pytest.mark.parametrize("species", SIZES)
def test_the_pivoted_factors_have_the_oracles_order_and_bits(gpu, tmp_path, species, warps):
    y = np.random.default_rng(1).standard_normal(species)
    with CudaSolver(isomers(tmp_path, species), gpu, warps=warps) as solver:
        for name, a in matrices(species):
            lu, dinv, order, x, _ = factored(solver, gpu, a, y, y, 0.0, True)
            with np.errstate(all="ignore"):
                ref_lu, ref_dinv, ref_order = oracle.dense_lu(a)
                ref_x = oracle.dense_solve(ref_lu, ref_dinv, ref_order, y)
            moved = ref_order != np.arange(species)
            assert not (name == "none" and moved.any()) and not (name == "exchanges" and species > 8 and not moved.any())
            if name == "far" and species > 8:  # rows that change their block of 8
                assert (ref_order // 8 != np.arange(species) // 8).any()
            assert np.array_equal(order, ref_order), name
            assert np.array_equal(lu, ref_lu, equal_nan=True) and np.array_equal(dinv, ref_dinv, equal_nan=True), name
            if np.isfinite(ref_lu).all():
                assert np.array_equal(x, ref_x, equal_nan=True), name
