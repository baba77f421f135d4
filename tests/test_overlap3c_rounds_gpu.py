"""3-center overlap of bases with f shells whose moments do not fit at once: several rounds
with a partial last one, and batches that end on a round's boundary.  Tiles are made cheap:
one element per species triple fills a tile of 32."""
import itertools

import numpy as np
import pytest
import torch

import aok_b200 as aok
import fakecuda
import oracle
from helpers import f32_round, rel_fro

W = aok.workloads
LS = [0, 0, 1, 1, 1, 2, 2, 3, 3]     # 43 functions
KEPT = 256 << 20                      # bytes of moments that a plan keeps


def moments(l):
    """Moments of a block: monomials r0^a r1^b r2^g h^d of degree l0 + l1 + l2 (h counts
    twice), each exponent bounded by the other two shells' momenta."""
    n = sum(l)
    return sum((n - a - b - g) % 2 == 0 and a + b + g <= n
               for a in range(l[1] + l[2] + 1) for b in range(l[0] + l[2] + 1) for g in range(l[0] + l[1] + 1))


TILE = sum(moments(t) for t in itertools.product(LS, repeat=3)) * 32 * 8
ROUND = KEPT // TILE


def test_rounds_of_a_call(tmp_path):
    """The launches of a call (device-less runtime): as many rounds as the count above says."""
    assert moments((0, 0, 0)) == 1 and moments((2, 2, 2)) == 41 and moments((3, 3, 3)) == 104
    body = f"""
out = []
for B in {[32 * (k * ROUND - 1) + d for k in (1, 2, 3) for d in (0, 1)]}:
    h = plan({LS}, 2, 1, 0, B)
    for repeat in range(2):                       # the first call sets up, with a launch of its own
        ops()
        assert L.aok_overlap3c(h, *[P(A)] * 9, I64(B), F64(1.0), P(0x77)) == 0
    k = [x[0] for x in ops()]
    out.append([sum("k_moments3" in x for x in k), sum("k_transform3" in x for x in k)])
    L.aok_plan_destroy(h)
print(json.dumps(out))
"""
    # ceil(B / 32) tiles and a partial one per species triple
    assert fakecuda.run(body, tmp_path) == [[1, 1], [2, 2], [2, 2], [3, 3], [3, 3], [4, 4]]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-6)])
@pytest.mark.parametrize("tiles", [2 * ROUND + 31, 2 * ROUND, 3 * ROUND + 1])
def test_several_rounds(dtype, tol, tiles):
    nsp, K = 6, 2
    rng = np.random.default_rng(61)
    r = f32_round if dtype == torch.float32 else np.asarray
    zeta = np.asfortranarray(r(np.exp(rng.uniform(-2, -0.5, (len(LS), 1, nsp))) * 2.5 ** np.arange(K)[None, :, None]))
    b = W.SpeciesBasis(ls=np.array(LS), zeta=zeta, D=np.asfortranarray(rng.uniform(0.1, 1.0, zeta.shape)),
                       nprim=np.full((len(LS), nsp), K), zlist=tuple(range(1, nsp + 1)))
    cob = aok.compile_basis(aok.orbitals_from_species_basis(b), dtype=dtype)
    assert ROUND < tiles <= nsp ** 3 and -(-tiles // ROUND) > 1
    # one element per species triple, so one tile each; two triples get a second element
    key = np.r_[rng.permutation(nsp ** 3)[:tiles], 0, 0]
    key[-2:] = key[:2]
    S = [key // nsp ** 2 + 1, key // nsp % nsp + 1, key % nsp + 1]
    pos = [np.asfortranarray(r(rng.standard_normal((3, len(key))))) for _ in range(3)]
    np_t = np.float32 if dtype == torch.float32 else np.float64
    V = aok.batch_overlap_3c(cob, *(aok.PStates(p.astype(np_t), s) for p, s in zip(pos, S)), FT=dtype, device_out=True)
    ref = oracle.overlap3c_orb(b.ls, cob.coef.cpu().numpy().astype(np.float64), zeta, *S, *pos, nthreads=8)
    got = V.cpu().numpy()
    for e in range(len(key)):
        assert rel_fro(got[..., e], ref[..., e]) < tol, e
