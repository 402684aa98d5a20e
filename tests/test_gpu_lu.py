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
