"""2-center overlap of batches with fewer tiles than the device holds (units of one panel of
a tile): partial tiles, several species pairs and the boundary between the two rules, against
the FP64 oracle at the tolerances of the other 2C tests, and bit for bit against the same
call on a plan of a large batch (whole tiles): both add an element's records in one order."""
import numpy as np
import pytest
import torch

import aok_b200 as aok
import oracle
from helpers import f32_round, rel_fro

W = aok.workloads
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-6)])
@pytest.mark.parametrize("nspecies", [1, 4])
def test_few_tiles(dtype, tol, nspecies):
    b = W.config2_basis(nspecies=nspecies)
    orb = aok.orbitals_from_species_basis(b)
    big = aok.compile_basis(orb, dtype=dtype)
    for B in (20001, 1, 31, 33, 257, 1500, 2400, 4700, 9500):
        pr = W.ragged_pairs(B, nspecies, 31)
        XA, XB = aok.PStates(pr.posA, list(pr.sidxA)), aok.PStates(pr.posB, list(pr.sidxB))
        whole = aok.batch_overlap(big, XA, XB, FT=dtype, device_out=True)
        if B > 10000:
            continue  # the plan is now one of a large batch
        S = aok.batch_overlap(aok.compile_basis(orb, dtype=dtype), XA, XB, FT=dtype, device_out=True)
        assert torch.equal(S, whole)
        r = f32_round if dtype == torch.float32 else np.asarray
        coef = r(oracle.compile_coef(r(b.zeta), r(b.D), b.ls))
        ref = oracle.overlap2c_orb(b.ls, coef, r(b.zeta), pr.sidxA, pr.sidxB, r(pr.posA), r(pr.posB), nthreads=8)
        assert rel_fro(S, ref) < tol
