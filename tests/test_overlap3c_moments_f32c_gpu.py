"""FP32C accuracy of the 3-center overlap of contracted bases with f shells, class by class:
moments and recursions are FP64, so an element is rounded to FP32 once where it is stored
(2^-24 of it at most, 2.5e-8 on average; up to 3.7e-8 where the aliased layout adds several)
and its exponentials, in FP32 up to d, are off by some 1e-7, which leaves less than 4e-8 of a
block's norm.  Together that is below 2^-24 for every class.  Sums and recursions in FP32 are
not: 8e-8 to 1.2e-7 from p-p-p on."""
import numpy as np
import pytest
import torch

import aok_b200 as aok
import oracle
from helpers import f32_round

W = aok.workloads
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,nspecies", [(2, 1), (3, 2), (8, 1)])
def test_error_of_every_class(K, nspecies):
    rng = np.random.default_rng(40 + K)
    ls = np.array([0, 1, 2, 3])
    zeta = f32_round(np.exp(rng.uniform(np.log(0.1), np.log(0.5), (4, 1, nspecies)))
                     * 2.5 ** np.arange(K)[None, :, None])
    b = W.SpeciesBasis(ls=ls, zeta=np.asfortranarray(zeta), D=np.asfortranarray(rng.uniform(0.1, 1.0, zeta.shape)),
                       nprim=np.full((4, nspecies), K), zlist=tuple(range(1, nspecies + 1)))
    cob = aok.compile_basis(aok.orbitals_from_species_basis(b), dtype=torch.float32)
    B = 200
    pos = [np.asfortranarray(f32_round(0.4 * rng.standard_normal((3, B)))) for _ in range(3)]
    pos[1][0] = f32_round(pos[1][0] + 1.2)
    pos[2][1] = f32_round(pos[2][1] + 1.0)
    S = [rng.integers(1, nspecies + 1, B) for _ in range(3)]
    V = aok.batch_overlap_3c(cob, *(aok.PStates(p.astype(np.float32), s) for p, s in zip(pos, S)), FT=torch.float32)
    ref = oracle.overlap3c_orb(ls, cob.coef.cpu().numpy().astype(np.float64), zeta, *S, *pos, nthreads=8)
    err = np.asarray(V, dtype=np.float64) - ref
    at = np.r_[0, np.cumsum((ls + 1) * (ls + 2) // 2)]
    sums = {}
    for a in range(4):
        for c in range(4):
            for d in range(4):
                k = tuple(sorted((ls[a], ls[c], ls[d]), reverse=True))
                box = np.s_[at[a]:at[a + 1], at[c]:at[c + 1], at[d]:at[d + 1]]
                e = sums.setdefault(k, np.zeros(2))
                e += [np.sum(err[box] ** 2), np.sum(ref[box] ** 2)]
    assert len(sums) == 20
    worst = {k: float(np.sqrt(e[0] / e[1])) for k, e in sums.items()}
    assert max(worst.values()) < 2.0 ** -24, worst
