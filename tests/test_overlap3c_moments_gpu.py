"""3-center overlap of bases with f shells (moments) at the sizes where it can go wrong:
partial tiles, every class up to f-f-f in every order of the centres, heavy blocks shared
by a CTA's warps, absent shells, element groups (blocks larger than the slab) with partial
tiles, and several rounds of moments.  Against the FP64 oracle at the tolerances of the
other 3C tests (FP64 1e-12, FP32C 2e-6)."""
import numpy as np
import pytest
import torch

import aok_b200 as aok
import oracle
from helpers import f32_round, rel_fro

W = aok.workloads
pytestmark = pytest.mark.gpu


def _run(b, B, dtype, seed, sample=None):
    rng = np.random.default_rng(seed)
    if dtype == torch.float32:
        b = W.SpeciesBasis(ls=b.ls, zeta=f32_round(b.zeta), D=b.D, nprim=b.nprim, zlist=b.zlist)
    cob = aok.compile_basis(aok.orbitals_from_species_basis(b), dtype=dtype)
    tr = W.config4_triples(B=B, seed=seed)
    pos = [f32_round(p) if dtype == torch.float32 else p for p in (tr.posA, tr.posB, tr.posC)]
    S = [rng.integers(1, b.NZ + 1, B) for _ in range(3)]
    V = aok.batch_overlap_3c(cob, *(aok.PStates(p.astype(np.float32) if dtype == torch.float32 else p, s)
                                    for p, s in zip(pos, S)), FT=dtype, device_out=True)
    at = np.arange(B) if sample is None else np.unique(np.r_[0:sample, B - sample:B, rng.integers(0, B, sample)])
    coef = cob.coef.cpu().numpy().astype(np.float64)
    ref = oracle.overlap3c_orb(b.ls, coef, b.zeta, *(s[at] for s in S), *(np.asfortranarray(p[:, at]) for p in pos),
                               nthreads=8)
    got = V[:, :, :, torch.as_tensor(at, device=V.device)]
    assert rel_fro(got, ref) < (1e-12 if dtype == torch.float64 else 2e-6)


def _basis(ls, K, seed, nspecies=1, nprim=None):
    rng = np.random.default_rng(seed)
    ns = len(ls)
    zeta = np.ones((ns, K, nspecies), order="F")
    D = np.zeros((ns, K, nspecies), order="F")
    n = np.full((ns, nspecies), K) if nprim is None else np.asarray(nprim)
    for s in range(ns):
        for g in range(nspecies):
            z0 = np.exp(rng.uniform(np.log(0.1), np.log(0.5)))
            zeta[s, :n[s, g], g] = z0 * 2.5 ** np.arange(n[s, g])
            D[s, :n[s, g], g] = rng.uniform(0.1, 1.0, n[s, g])
    return W.SpeciesBasis(ls=np.asarray(ls, dtype=np.int64), zeta=zeta, D=D, nprim=n, zlist=tuple(range(1, nspecies + 1)))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("K,B", [(2, 1), (3, 33)])
def test_every_class_up_to_f(dtype, K, B):
    _run(_basis([0, 1, 2, 3], K, 11), B, dtype, 21)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("B", [31, 71])
def test_heavy_blocks_and_absent_shells(dtype, B):
    b = _basis([0, 0, 1, 2, 3], 9, 12, 2, [[9, 8], [0, 3], [7, 9], [9, 0], [1, 2]])
    _run(b, B, dtype, 22)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_heavy_f_blocks(dtype):
    _run(_basis([0, 3], 5, 13), 40, dtype, 23)


def test_several_rounds_of_moments():
    # 45 functions: more tiles than the kept moments hold at once
    _run(_basis([0, 0, 1, 1, 1, 2, 2, 3, 3], 2, 15), 900, torch.float64, 25, sample=6)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_few_primitives_and_both_paths_on_one_plan(dtype):
    # 1.3 triples per function on average (explicit tables), 8.6 (moments), then 1.3 again
    few = _basis([0, 0, 1, 2, 3], 3, 17, nprim=[[3], [1], [1], [1], [1]])
    many = _basis([0, 0, 1, 2, 3], 3, 18, nprim=[[2], [3], [2], [2], [2]])
    for b in (few, many, few):
        _run(b, 45, dtype, 27)
