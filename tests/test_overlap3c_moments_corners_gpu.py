"""3-center overlap through moments at the edges of its inputs: infinite and NaN positions
(the same elements are NaN as with explicit E tables) and a length scale."""
import numpy as np
import pytest
import torch

import aok_b200 as aok
from aok_b200 import _dev, _lib

W = aok.workloads
pytestmark = pytest.mark.gpu
LS = [0, 0, 1, 2, 3]


def _call(nprim, pos, dtype, lengthscale=1.0, nspecies=1):
    """Blocks (B, N, N, N) of a basis with the given primitives per shell on its own plan."""
    rng = np.random.default_rng(71)
    K, ns, B = 3, len(LS), pos[0].shape[1]
    zeta = np.ones((ns, K, nspecies), order="F")
    coef = np.zeros((ns, K, nspecies), order="F")
    for s in range(ns):
        zeta[s, :nprim[s]] = 0.3 * 2.5 ** np.arange(nprim[s])[:, None]
        coef[s, :nprim[s]] = rng.uniform(0.1, 1.0, (nprim[s], nspecies))
    L = _lib.load()
    plan = _dev.Plan(LS, K, nspecies, _dev.prec_of(dtype), B)
    N = 1 + 1 + 3 + 6 + 10
    out = torch.zeros((B, N, N, N), dtype=dtype, device="cuda")
    dev = [_dev.to_colmajor(x, dtype) for x in (zeta, coef, *pos)]
    S = [torch.as_tensor(rng.integers(1, nspecies + 1, B)).cuda() for _ in range(3)]
    _lib.check(L.aok_overlap3c(plan.h, _dev.ctypes.c_void_p(out.data_ptr()), *(_dev.ptr(x) for x in dev),
                               *(_dev.ctypes.c_void_p(s.data_ptr()) for s in S), B, lengthscale, _dev.stream()))
    return out


FEW, MANY = (3, 1, 1, 1, 1), (3, 2, 2, 2, 2)      # explicit tables, moments


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_positions_that_are_not_finite(dtype):
    rng = np.random.default_rng(72)
    B = 70
    pos = [np.asfortranarray(rng.standard_normal((3, B))) for _ in range(3)]
    e = 0
    for bad in (np.inf, -np.inf, np.nan):
        for c in range(3):
            for x in range(3):
                pos[c][x, e] = bad
                e += 1
        for x in range(3):                        # two centres: their difference is NaN
            pos[0][x, e] = pos[1][x, e] = bad
            e += 1
    tables, moments = _call(FEW, pos, dtype), _call(MANY, pos, dtype)
    assert torch.equal(torch.isnan(moments), torch.isnan(tables))
    assert not torch.isinf(moments).any()
    assert torch.isnan(moments[:e]).any(dim=(1, 2, 3)).all() and torch.isfinite(moments[e:]).all()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nspecies", [1, 2])
def test_lengthscale(dtype, nspecies):
    rng = np.random.default_rng(73)
    f = np.float32 if dtype == torch.float32 else np.float64
    pos = [np.asfortranarray(rng.standard_normal((3, 77)).astype(f)) for _ in range(3)]
    scaled = _call(MANY, pos, dtype, 1.7, nspecies)
    assert torch.equal(scaled, _call(MANY, [p * f(1.7) for p in pos], dtype, 1.0, nspecies))
    assert not torch.equal(scaled, _call(MANY, pos, dtype, 1.0, nspecies))
