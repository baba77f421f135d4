"""2-center overlap of few tiles (units of one panel of a tile, narrow panels) against the
same pairs inside a batch of whole tiles on a plan with wide panels: bit for bit, since an
element's records are added in one order whatever the panels are."""
import numpy as np
import pytest
import torch

import aok_b200 as aok
import fakecuda
from aok_b200 import _dev, _lib

W = aok.workloads
BIG = 20001
SPLIT = {torch.float64: (1, 33, 257, 1500, 2400), torch.float32: (1, 33, 1000, 2400, 4700)}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_which_batches_are_split(tmp_path, dtype):
    b = W.config2_basis()
    body = f"""
out = []
for B in {list(SPLIT[dtype]) + [BIG]}:
    h = plan({[int(l) for l in b.ls]}, {b.K}, {b.NZ}, {_dev.prec_of(dtype)}, B)
    ops()
    assert L.aok_overlap2c(h, *[P(A)] * 7, I64(B), F64(1.0), P(0x77)) == 0
    out += [x[0] for x in ops() if "k_overlap2cI" in x[0]]
    L.aok_plan_destroy(h)
print(json.dumps(out))
"""
    names = fakecuda.run(body, tmp_path)          # the last template argument: split
    assert ["Lb1E" in k for k in names] == [True] * len(SPLIT[dtype]) + [False]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nspecies", [1, 4])
def test_split_equals_whole_tiles(dtype, nspecies):
    L = _lib.load()
    b = W.config2_basis(nspecies=nspecies)
    pr = W.ragged_pairs(BIG, nspecies, 37)
    N = b.nbf_total
    zeta, D = _dev.to_colmajor(b.zeta, dtype), _dev.to_colmajor(b.D, dtype)
    coef = _dev.colmajor_empty(b.zeta.shape, dtype)
    pos = [_dev.to_colmajor(p, dtype) for p in (pr.posA, pr.posB)]
    sidx = [torch.as_tensor(np.ascontiguousarray(s)).cuda() for s in (pr.sidxA, pr.sidxB)]

    def run(plan, B, fixed):
        out = _dev.colmajor_empty((N, N, B), dtype)
        out.fill_(float("nan"))
        if fixed:
            _lib.check(L.aok_plan_set_basis(plan.h, _dev.ptr(zeta), _dev.ptr(coef), _dev.stream()))
        par = (None, None) if fixed else (_dev.ptr(zeta), _dev.ptr(coef))
        _lib.check(L.aok_overlap2c(plan.h, _dev.ptr(out), *par, *(_dev.ptr(p) for p in pos),
                                   *(_dev.ctypes.c_void_p(s.data_ptr()) for s in sidx), B, 1.0, _dev.stream()))
        return out

    big = _dev.Plan(b.ls, b.K, b.NZ, _dev.prec_of(dtype), BIG)
    _lib.check(L.aok_compile_coef(big.h, _dev.ptr(coef), _dev.ptr(zeta), _dev.ptr(D), _dev.stream()))
    whole = run(big, BIG, True)
    for B in SPLIT[dtype]:
        small = _dev.Plan(b.ls, b.K, b.NZ, _dev.prec_of(dtype), B)
        for plan in (small, big):                 # narrow panels, wide panels
            for fixed in (True, False):
                assert torch.equal(run(plan, B, fixed), whole[:, :, :B]), (B, plan is small, fixed)
