"""The calls whose first kernel is launched programmatically, captured into a CUDA graph right
after work on another stream was joined, two in a row: replays give the bits of eager calls."""
import ctypes

import numpy as np
import pytest
import torch

import aok_b200 as aok
from aok_b200 import _dev, _lib

W = aok.workloads
pytestmark = pytest.mark.gpu


def p(t):
    return ctypes.c_void_p(t.data_ptr())


def _pairs(FT, B, n):
    b = W.config2_basis(nspecies=2)
    rng = np.random.default_rng(81)
    par = [_dev.to_colmajor(x, FT) for x in (b.zeta, b.D)]
    pos = [torch.as_tensor(rng.standard_normal((B, 3))).to("cuda", FT) for _ in range(n)]
    sp = [torch.as_tensor(rng.integers(1, 3, B)).cuda() for _ in range(n)]
    return b, par, pos, sp, _dev.Plan(b.ls, b.K, b.NZ, _dev.prec_of(FT), B)


def gradient(FT, B=300):
    b, par, pos, sp, plan = _pairs(FT, B, 2)
    N, L = b.nbf_total, _lib.load()
    out = [torch.empty((B, N, N), dtype=FT, device="cuda")] + [_dev.colmajor_empty(b.zeta.shape, FT) for _ in range(2)]
    ct = torch.as_tensor(np.random.default_rng(82).standard_normal((B, N, N))).to("cuda", FT)

    def call():
        geo = (*map(_dev.ptr, par), *map(p, pos), *map(p, sp), B, 1.0, _dev.stream())
        _lib.check(L.aok_overlap2c_rrule(plan.h, p(out[0]), *geo))
        _lib.check(L.aok_overlap_pullback_ps_rrule(plan.h, _dev.ptr(out[1]), _dev.ptr(out[2]), p(ct), *geo))
    return call, out


def overlap3c(FT, B=100):
    b, par, pos, sp, plan = _pairs(FT, B, 3)
    N, L = b.nbf_total, _lib.load()
    out = [torch.empty((B, N, N, N), dtype=FT, device="cuda")]

    def call():
        _lib.check(L.aok_overlap3c(plan.h, p(out[0]), *map(_dev.ptr, par), *map(p, pos), *map(p, sp), B, 1.0,
                                   _dev.stream()))
    return call, out


def overlap3c_gb(FT, B=100):
    rng = np.random.default_rng(83)
    ls, K, L = [0, 1, 2, 3], 2, _lib.load()
    plan = _dev.Plan(ls, K, 1, _dev.prec_of(FT), B)
    nprim = torch.full((4,), K, dtype=torch.int64, device="cuda")
    off = torch.arange(0, 4 * K, K, dtype=torch.int64, device="cuda")
    flat = [torch.as_tensor(x).to("cuda", FT) for x in (rng.uniform(0.1, 1, 4 * K), rng.uniform(0.2, 2, 4 * K))]
    pos = [torch.as_tensor(rng.standard_normal((B, 3))).to("cuda", FT) for _ in range(3)]
    out = [torch.empty((B, 20, 20, 20), dtype=FT, device="cuda")]

    def call():
        _lib.check(L.aok_overlap3c_gb(plan.h, p(out[0]), p(nprim), p(off), *map(p, flat), *map(p, pos), B,
                                      _dev.stream()))
    return call, out


def evaluate(FT, nX=3000):
    b = W.config1_basis()
    orb = aok.orbitals_from_species_basis(b)
    X, s = W.config1_points(nX=nX, seed=84)
    L = _lib.load()
    plan = _dev.orb_plan_for(b.zeta.shape[0], b.K, b.NZ, orb.Rnl.powers(), orb.radidx, orb.ylmidx, orb.L,
                             orb.Rnl.kind, _dev.prec_of(FT))
    X, zeta, D = (_dev.to_colmajor(x, FT) for x in (X, b.zeta, b.D))
    s = torch.as_tensor(s).cuda()
    dP = _dev.to_colmajor(np.random.default_rng(85).standard_normal((nX, len(orb))), FT)
    out = [_dev.colmajor_empty((nX, len(orb)), FT), _dev.colmajor_empty((3, nX), FT)]
    out += [_dev.colmajor_empty(b.zeta.shape, FT) for _ in range(2)]

    def call():
        arg = (_dev.ptr(X), p(s), _dev.ptr(zeta), _dev.ptr(D), nX, 1.0, _dev.stream())
        _lib.check(L.aok_evaluate(plan.h, _dev.ptr(out[0]), *arg))
        _lib.check(L.aok_evaluate_pullback(plan.h, *map(_dev.ptr, out[1:]), _dev.ptr(dP), *arg))
    return call, out


@pytest.mark.parametrize("make", [gradient, overlap3c, overlap3c_gb, evaluate])
@pytest.mark.parametrize("FT", [torch.float64, torch.float32])
def test_captured_calls_equal_eager_ones(make, FT):
    call, out = make(FT)
    call()
    torch.cuda.synchronize()
    want = [o.clone() for o in out]
    work, other = torch.cuda.Stream(), torch.cuda.Stream()
    a, c = torch.zeros(1000, device="cuda"), torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=work, capture_error_mode="thread_local"):
        a.add_(1)
        other.wait_stream(work)
        with torch.cuda.stream(other):
            c.add_(2)
        work.wait_stream(other)
        call()
        call()
        a.add_(c)
    for _ in range(2):
        for o in out:
            o.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o, w in zip(out, want))
    assert a[0].item() == 8 and c[0].item() == 4   # 1 + 2, then + 1 + 4
    del g
