"""Performance cases: the calls that a program using this library makes, with their
inputs, one pass each, the work a pass cannot do without, and FP64 results in plain torch.

The device-resident path is the C interface (include/aok.h), as a host framework that owns
its arrays calls it; one case goes through the Python package with host inputs.  Bases are
the synthetic ones of aok_b200.workloads (shell structure from `basis_seed`), with exponents
and coefficients varied by the seed; geometries and species are drawn from the seed.

Kinds:
  overlap2c      2-center overlap of a species-aware compiled basis (records fixed once)
  overlap2c_gb   2-center overlap on the GaussianBasis path (parameters given per call)
  overlap2c_api  aok.batch_overlap_ on host PState batches (Python package)
  gradient       (zeta, D) gradient step of an overlap loss: rrule forward + its pullback
  position       position pullback of the 2-center overlap
  evaluate_ed    orbital values and spatial gradients
  evaluate_step  orbital values, then the pullback to positions and (zeta, D)
  overlap3c_gb   3-center overlap on the GaussianBasis path
  overlap3c      3-center overlap of a species-aware basis
"""
import ctypes
import math

import numpy as np
import torch

import aok_b200 as aok
from aok_b200 import _dev, _lib

MAX_OUT_BYTES = 330e6  # the largest output of a listed case (65,536 blocks of 35 x 35 in FP32)


# --------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------


def listed():
    return [
        # A pair list of a mid-size molecular data set, four elements, contracted s-f shells:
        # the library's headline workload, single-precision storage.
        dict(name="overlap2c-f32-65536", kind="overlap2c", basis="mixed", dtype="f32", B=65536, basis_seed=1002),
        # The same in double precision (reference-quality integrals), an odd batch.
        dict(name="overlap2c-f64-20011", kind="overlap2c", basis="mixed", dtype="f64", B=20011, basis_seed=1002),
        # Uncontracted (one primitive per shell) basis, as in fitted or even-tempered sets.
        dict(name="overlap2c-k1-f32-40961", kind="overlap2c", basis="k1", dtype="f32", B=40961, basis_seed=1005),
        # A short dimer scan with one element: the smallest calls, parameters passed each time.
        dict(name="overlap2c-gb-f64-257", kind="overlap2c_gb", basis="small", dtype="f64", B=257, basis_seed=1000),
        # The Python package on host data: a few hundred pairs per call from an MD frame.
        dict(name="overlap2c-api-f64-500", kind="overlap2c_api", basis="mixed", dtype="f64", B=500, basis_seed=1002),
        # One step of fitting (zeta, D) to target overlaps by a squared residual.
        dict(name="gradient-f32-16384", kind="gradient", loss="residual", basis="mixed", dtype="f32", B=16384,
             basis_seed=1002),
        # A small fitting batch in double precision, the cotangent given by the caller's loss.
        dict(name="gradient-f64-3001", kind="gradient", loss="cotangent", basis="mixed", dtype="f64", B=3001,
             basis_seed=1002),
        # Forces from an overlap-dependent energy.
        dict(name="position-f32-8191", kind="position", basis="mixed", dtype="f32", B=8191, basis_seed=1002),
        # Orbitals and their gradients on a large integration grid.
        dict(name="evaluate_ed-f32-1048576", kind="evaluate_ed", basis="small", species=3, radial="gaussian",
             dtype="f32", nX=1 << 20, basis_seed=1001),
        # One training pass of an orbital layer over a grid batch.
        dict(name="evaluate_step-f32-262144", kind="evaluate_step", basis="small", species=3, radial="gaussian",
             dtype="f32", nX=1 << 18, basis_seed=1001),
        # Three-center overlaps of a small one-element basis over many triples.
        dict(name="overlap3c-gb-f32-4096", kind="overlap3c_gb", basis="small", dtype="f32", B=4096, basis_seed=1000),
        # Three-center overlaps of two elements with shells up to f, double precision.
        dict(name="overlap3c-f64-777", kind="overlap3c", basis="mixed", species=2, dtype="f64", B=777,
             basis_seed=1002),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["overlap2c", "overlap2c", "overlap2c_gb", "overlap2c_api", "gradient", "gradient", "position",
                       "evaluate_ed", "evaluate_step", "overlap3c_gb", "overlap3c"])
    c = dict(kind=kind, dtype=rng.choice(["f32", "f64"]), basis_seed=rng.randrange(2000, 100000))
    if kind in ("evaluate_ed", "evaluate_step"):
        c.update(basis="small", species=rng.randint(1, 4), radial=rng.choice(["gaussian", "gaussian", "slater"]))
        c["nX"] = _log_int(rng, 1000, (1 << 20) if kind == "evaluate_ed" else (1 << 18))
        if c["dtype"] == "f64":
            c["nX"] //= 2
        return c
    if kind == "gradient":
        c["loss"] = rng.choice(["residual", "cotangent"])
    if kind in ("overlap2c_gb", "overlap3c_gb"):
        c["basis"] = rng.choice(["small", "single"])
    elif kind == "overlap2c":
        c["basis"] = rng.choice(["mixed", "mixed", "k1"])
    elif kind == "overlap3c":
        c.update(basis=rng.choice(["small", "mixed"]), species=2)
    else:
        c["basis"] = "mixed"
    lo, hi = {"overlap2c": (1000, 65536), "overlap2c_gb": (200, 65536), "overlap2c_api": (100, 1000),
              "gradient": (1000, 16384), "position": (1000, 16384), "overlap3c_gb": (100, 4096),
              "overlap3c": (50, 1500)}[kind]
    b = _basis(c)
    esz = 8 if c["dtype"] == "f64" else 4
    n = b.nbf_total ** (3 if kind.startswith("overlap3c") else 2)
    if kind == "gradient":
        n *= 4  # residual: S, its target, and the FP64 side's cost
    c["B"] = _log_int(rng, lo, max(lo + 1, min(hi, int(0.8 * MAX_OUT_BYTES / (n * esz)))))
    return c


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------


def _basis(case):
    """The case's shell structure and primitive counts (zeta, D: its unvaried parameters)."""
    W, s, kind = aok.workloads, case["basis_seed"], case["basis"]
    if kind == "mixed":
        return W.config2_basis(seed=s, nspecies=case.get("species", 4))
    if kind == "single":
        return W.config2_basis(seed=s, nspecies=1)
    if kind == "k1":
        return W.outputbound_basis(seed=s)
    return W.config0_basis(seed=s, nspecies=case.get("species", 1))


def _ft(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _host_rng(case, seed):
    return np.random.default_rng([int(seed), case["basis_seed"]])


def _params(b, rng, amount=0.05):
    """Varied (zeta, D) on the real slots; padding keeps (1, 0).  Float64, (ns, K, NZ)."""
    real = b.D != 0
    z = np.where(real, b.zeta * np.exp(amount * rng.standard_normal(b.zeta.shape)), b.zeta)
    D = np.where(real, b.D * (1.0 + amount * rng.standard_normal(b.D.shape)), b.D)
    return z, D


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _pairs(case, b, seed):
    """Species-ragged pairs at 0.5 to 8 bohr in random directions, on the device."""
    g, B, FT = _gen(seed), case["B"], _ft(case)
    kw = dict(generator=g, device="cuda", dtype=torch.float64)
    A = 0.4 * torch.randn((B, 3), **kw)
    u = torch.randn((B, 3), **kw)
    d = 0.5 + 7.5 * torch.rand((B, 1), **kw)
    Bp = A + d * u / u.norm(dim=1, keepdim=True)
    sA = torch.randint(1, b.NZ + 1, (B,), generator=g, device="cuda")
    sB = torch.randint(1, b.NZ + 1, (B,), generator=g, device="cuda")
    return A.to(FT).contiguous(), Bp.to(FT).contiguous(), sA, sB


def _triples(case, b, seed):
    """Bonded triples: B near (1.2, 0, 0) and C near (0, 1, 0) from A, each moved by 0.4 bohr."""
    g, B, FT = _gen(seed), case["B"], _ft(case)
    X = [0.4 * torch.randn((B, 3), generator=g, device="cuda", dtype=torch.float64) for _ in range(3)]
    X[1][:, 0] += 1.2
    X[2][:, 1] += 1.0
    S = [torch.randint(1, b.NZ + 1, (B,), generator=g, device="cuda") for _ in range(3)]
    return [x.to(FT).contiguous() for x in X], S


def _dev_cm(a, FT):
    """(n1, ..., nk) host array -> the device memory of its column-major layout."""
    return torch.as_tensor(np.ascontiguousarray(np.asarray(a).transpose())).to("cuda", FT)


def _norms(ls, z, D):
    """sqrt of the Cartesian self-overlap of each contraction, (ns, NZ)."""
    out = np.zeros((z.shape[0], z.shape[2]))
    for s, l in enumerate(ls):
        c = math.pi ** 1.5 * math.prod(range(2 * int(l) - 1, 0, -2)) / 2.0 ** int(l)
        zz = z[s][:, None, :] + z[s][None, :, :]
        out[s] = np.sqrt(c * (D[s][:, None, :] * D[s][None, :, :] / zz ** (l + 1.5)).sum(axis=(0, 1)))
    return out


def _gb_arrays(b, z, D):
    """Flat tables of the first species: shells present, their primitive counts, coef, alpha."""
    keep = np.flatnonzero(b.nprim[:, 0] > 0)
    nprim = b.nprim[keep, 0]
    nrm = _norms(b.ls, z, D)
    alpha = np.concatenate([z[s, :n, 0] for s, n in zip(keep, nprim)])
    coef = np.concatenate([D[s, :n, 0] / nrm[s, 0] for s, n in zip(keep, nprim)])
    return b.ls[keep], nprim, coef, alpha


def _new_plan(ls, K, NZ, FT, B):
    return _dev.Plan(ls, int(K), int(NZ), _dev.prec_of(FT), int(B))


def _spec(b):
    """Radial -> orbital maps of a shared (n, l) structure."""
    s = aok.workloads.orbital_spec(b.ls)
    return s.iR, s.iY, s.L


def _points(case, b, seed):
    g, n, FT = _gen(seed), case["nX"], _ft(case)
    X = 2.0 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return X.to(FT).contiguous(), torch.randint(1, b.NZ + 1, (n,), generator=g, device="cuda")


def _poly(case, b):
    """Radial powers: none for Gaussians; n - 1 of the n-th shell of its l for Slater radials."""
    if case["radial"] == "gaussian":
        return [0] * b.nshells
    seen, out = {}, []
    for l in b.ls:
        seen[int(l)] = seen.get(int(l), 0) + 1
        out.append(seen[int(l)] - 1)
    return out


def _overlap_inputs(case, seed):
    """Everything the overlap paths are given: basis, (zeta, D) at the element type, geometry."""
    b, FT = _basis(case), _ft(case)
    z, D = _params(b, _host_rng(case, seed))
    if FT == torch.float32:
        z, D = z.astype(np.float32).astype(np.float64), D.astype(np.float32).astype(np.float64)
    return b, FT, z, D


def _target(case, seed, b, z, D, geo):
    """Overlaps of perturbed parameters, the data a residual loss is fitted to."""
    rng = _host_rng(case, seed + 1)
    real = b.D != 0
    zt = np.where(real, z * np.exp(0.1 * rng.standard_normal(z.shape)), z)
    Dt = np.where(real, D + 0.05 * rng.standard_normal(D.shape), D)
    z64, D64 = (torch.as_tensor(a, device="cuda") for a in (zt, Dt))
    return _overlap2c_64(b.ls, z64, _coef_64(b.ls, z64, D64), *geo).to(_ft(case))


def _cotangent(case, seed, shape):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 31 + 5)
    return torch.randn(shape, generator=g, device="cuda", dtype=_ft(case))


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "L": _lib.load()}
    if kind in ("evaluate_ed", "evaluate_step"):
        b, FT, z, D = _overlap_inputs(case, seed)
        iR, iY, L = _spec(b)
        X, sidx = _points(case, b, seed)
        n, nOrb = case["nX"], len(iR)
        st.update(X=X, sidx=sidx, zeta=_dev_cm(z, FT), D=_dev_cm(D, FT), n=n,
                  plan=_dev.OrbPlan(b.nshells, b.K, b.NZ, _poly(case, b), iR, iY, L,
                                    _lib.AOK_RADIAL_SLATER if case["radial"] == "slater" else _lib.AOK_RADIAL_GAUSSIAN,
                                    _dev.prec_of(FT)),
                  P=torch.empty((nOrb, n), dtype=FT, device="cuda"))
        if kind == "evaluate_ed":
            st["dP"] = torch.empty((nOrb, n, 3), dtype=FT, device="cuda")
        else:
            st.update(ct=_cotangent(case, seed, (nOrb, n)), dX=torch.empty_like(X), dz=torch.empty_like(st["zeta"]),
                      dD=torch.empty_like(st["D"]))
        return st
    b, FT, z, D = _overlap_inputs(case, seed)
    B = case["B"]
    st["B"] = B
    if kind in ("overlap2c_gb", "overlap3c_gb"):
        ls, nprim, coef, alpha = _gb_arrays(b, z, D)
        N = int(((ls + 1) * (ls + 2) // 2).sum())
        X, _ = _triples(case, b, seed)
        if kind == "overlap2c_gb":
            X = X[:2]
        st.update(plan=_new_plan(ls, nprim.max(), 1, FT, B), X=X, nprim=torch.as_tensor(nprim).cuda(),
                  off=torch.as_tensor(np.concatenate([[0], np.cumsum(nprim)])).cuda(),
                  coef=torch.as_tensor(coef).to("cuda", FT), alpha=torch.as_tensor(alpha).to("cuda", FT),
                  out=torch.empty((B,) + (N,) * len(X), dtype=FT, device="cuda"))
        return st
    N = b.nbf_total
    if kind == "overlap3c":
        X, S = _triples(case, b, seed)
        shape = (B, N, N, N)
    else:
        *X, sA, sB = _pairs(case, b, seed)
        S = [sA, sB]
        shape = (B, N, N)
    if kind == "overlap2c_api":
        zl = (1, 6, 7, 8)[:b.NZ]
        sb = aok.workloads.SpeciesBasis(ls=b.ls, zeta=z, D=D, nprim=b.nprim, zlist=zl)
        cob = aok.compile_basis(aok.orbitals_from_species_basis(sb, "bohr"), dtype=FT)
        lab = np.asarray(zl)
        st.update(cob=cob, out=torch.empty(shape, dtype=FT, device="cuda"),
                  A=aok.PStates(X[0].cpu().numpy().T, lab[S[0].cpu().numpy() - 1]),
                  Bs=aok.PStates(X[1].cpu().numpy().T, lab[S[1].cpu().numpy() - 1]))
        return st
    plan = _new_plan(b.ls, b.K, b.NZ, FT, B)
    zd, Dd = _dev_cm(z, FT), _dev_cm(D, FT)
    st.update(plan=plan, X=X, S=S, zeta=zd, D=Dd)
    if kind == "gradient":
        st.update(loss=case["loss"], out=torch.empty(shape, dtype=FT, device="cuda"), dz=torch.empty_like(zd),
                  dD=torch.empty_like(Dd))
        st["ct"] = (_target(case, seed, b, z, D, (*X, *S)) if case["loss"] == "residual"
                    else _cotangent(case, seed, shape))
        return st
    coef = torch.empty_like(zd)
    _lib.check(st["L"].aok_compile_coef(plan.h, _p(coef), _p(zd), _p(Dd), _dev.stream()))
    st["coef"] = coef
    if kind == "position":
        st.update(ct=_cotangent(case, seed, shape), dA=torch.empty_like(X[0]), dB=torch.empty_like(X[1]))
    else:
        st["out"] = torch.empty(shape, dtype=FT, device="cuda")
    if kind == "overlap2c":  # the compiled basis: its records are fixed once
        _lib.check(st["L"].aok_plan_set_basis(plan.h, _p(zd), _p(coef), _dev.stream()))
    return st


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def run(st):
    kind, L = st["kind"], st["L"]
    if kind == "overlap2c_api":
        aok.batch_overlap_(st["out"].permute(2, 1, 0), st["cob"], st["A"], st["Bs"])
        return st["out"]
    h, stream = st["plan"].h, _dev.stream()
    if kind == "evaluate_ed":
        _lib.check(L.aok_evaluate_ed(h, _p(st["P"]), _p(st["dP"]), _p(st["X"]), _p(st["sidx"]), _p(st["zeta"]),
                                     _p(st["D"]), st["n"], 1.0, stream))
        return st["P"], st["dP"]
    if kind == "evaluate_step":
        _lib.check(L.aok_evaluate(h, _p(st["P"]), _p(st["X"]), _p(st["sidx"]), _p(st["zeta"]), _p(st["D"]), st["n"],
                                  1.0, stream))
        _lib.check(L.aok_evaluate_pullback(h, _p(st["dX"]), _p(st["dz"]), _p(st["dD"]), _p(st["ct"]), _p(st["X"]),
                                           _p(st["sidx"]), _p(st["zeta"]), _p(st["D"]), st["n"], 1.0, stream))
        return st["P"], st["dX"], st["dz"], st["dD"]
    X = [_p(x) for x in st["X"]]
    if kind in ("overlap2c_gb", "overlap3c_gb"):
        call = L.aok_overlap2c_gb if kind == "overlap2c_gb" else L.aok_overlap3c_gb
        _lib.check(call(h, _p(st["out"]), _p(st["nprim"]), _p(st["off"]), _p(st["coef"]), _p(st["alpha"]), *X,
                        st["B"], stream))
        return st["out"]
    geo = X + [_p(s) for s in st["S"]] + [st["B"], 1.0, stream]
    if kind == "overlap2c":
        _lib.check(L.aok_overlap2c(h, _p(st["out"]), None, None, *geo))
        return st["out"]
    if kind == "overlap3c":
        _lib.check(L.aok_overlap3c(h, _p(st["out"]), _p(st["zeta"]), _p(st["coef"]), *geo))
        return st["out"]
    if kind == "position":
        _lib.check(L.aok_overlap2c_position_pullback(h, _p(st["dA"]), _p(st["dB"]), _p(st["ct"]), _p(st["zeta"]),
                                                     _p(st["coef"]), *geo))
        return st["dA"], st["dB"]
    par = [_p(st["zeta"]), _p(st["D"])]
    _lib.check(L.aok_overlap2c_rrule(h, _p(st["out"]), *par, *geo))
    if st["loss"] == "residual":
        _lib.check(L.aok_overlap_pullback_ps_rrule_residual(h, _p(st["dz"]), _p(st["dD"]), _p(st["out"]),
                                                            _p(st["ct"]), 2.0, *par, *geo))
    else:
        _lib.check(L.aok_overlap_pullback_ps_rrule(h, _p(st["dz"]), _p(st["dD"]), _p(st["ct"]), *par, *geo))
    return st["out"], st["dz"], st["dD"]


# --------------------------------------------------------------------------
# Work of one pass
# --------------------------------------------------------------------------


def _mean_counts(b):
    """Mean primitive count per shell over the species drawn uniformly."""
    return b.nprim.mean(axis=1)


def work(case):
    b = _basis(case)
    esz = 8 if case["dtype"] == "f64" else 4
    kind = case["kind"]
    if kind in ("evaluate_ed", "evaluate_step"):
        n, nOrb = case["nX"], len(_spec(b)[0])
        prims = float(_mean_counts(b).sum())
        point = 3 * esz + 8 + nOrb * esz
        flops = 8 * prims + 60 + 2 * nOrb
        if kind == "evaluate_ed":
            return {"bytes": n * (point + 3 * nOrb * esz), "flops": n * (flops + 12 * nOrb + 4 * prims)}
        return {"bytes": n * (point + nOrb * esz + 3 * esz), "flops": n * (2 * flops + 12 * nOrb + 8 * prims)}
    ls, B = b.ls, case["B"]
    K = _mean_counts(b)
    if kind in ("overlap2c_gb", "overlap3c_gb"):
        ls, K = ls[b.nprim[:, 0] > 0], b.nprim[b.nprim[:, 0] > 0, 0]
    nc = (ls + 1) * (ls + 2) // 2
    N = int(nc.sum())
    k1, c1 = float(K.sum()), float((K > 0) @ nc)
    slots = float((K * (ls + 1)).sum())
    if kind in ("overlap3c", "overlap3c_gb"):
        # per primitive triple: exponent and prefactor; per product of powers: one table entry and axis
        flops = 20 * k1 ** 3 + 15 * slots ** 3 / 3 + 3 * c1 ** 3
        return {"bytes": B * (N ** 3 * esz + 3 * (3 * esz + (0 if kind.endswith("gb") else 8))), "flops": B * flops}
    # per primitive pair: exponent; per moment slot: one multiply-add; per output: its geometry terms
    flops = 10 * k1 ** 2 + slots ** 2 + 6 * c1 ** 2
    geo = 2 * (3 * esz + (0 if kind == "overlap2c_gb" else 8))
    if kind == "gradient":
        return {"bytes": B * (3 * N * N * esz + geo) if case["loss"] == "residual" else B * (2 * N * N * esz + geo),
                "flops": 4 * B * flops}
    if kind == "position":
        return {"bytes": B * (N * N * esz + geo + 6 * esz), "flops": 2 * B * flops}
    return {"bytes": B * (N * N * esz + geo), "flops": B * flops}


# --------------------------------------------------------------------------
# FP64 results in plain torch
# --------------------------------------------------------------------------


def _cart(l):
    """Cartesian powers of a shell: x descending, then z ascending."""
    return [(x, l - x - zz, zz) for x in range(l, -1, -1) for zz in range(0, l - x + 1)]


def _coef_64(ls, z, D):
    """D over the Cartesian norm of its contraction; 0 for a shell absent from a species."""
    rows = []
    for s, l in enumerate(ls):
        l = int(l)
        c = math.pi ** 1.5 * math.prod(range(2 * l - 1, 0, -2)) / 2.0 ** l
        zz = z[s][:, None, :] + z[s][None, :, :]
        n = c * (D[s][:, None, :] * D[s][None, :, :] / zz ** (l + 1.5)).sum(dim=(0, 1))
        here = n > 0
        rows.append(torch.where(here, D[s] / torch.where(here, n, torch.ones_like(n)).sqrt(), torch.zeros_like(D[s])))
    return torch.stack(rows)


def _grow(T, ls, shifts, h):
    """1-D overlap tables T[powers] from T[0, ..] = 1 by the Obara-Saika recursion; every
    entry is (3, n, P).  Returns them stacked (prod(l + 1), 3, n, P), last power fastest."""
    idx = [()]
    for l in ls:
        idx = [i + (k,) for i in idx for k in range(l + 1)]
    for i in idx:
        if sum(i) == 0:
            continue
        a = next(k for k in range(len(ls)) if i[k])
        low = i[:a] + (i[a] - 1,) + i[a + 1:]
        v = shifts[a] * T[low]
        for k in range(len(ls)):
            if low[k]:
                v = v + (low[k] * h) * T[low[:k] + (low[k] - 1,) + low[k + 1:]]
        T[i] = v
    return torch.stack([T[i] for i in idx])


def _block_64(ls, E, w, n):
    """Contracted block, flattened in output order (first index fastest): component products of
    the tables times the weights w (n, P), summed over P; a component goes to
    c1 + (2 l1 + 1) c2 + (2 l1 + 1)(2 l2 + 1) c3, several to one element from d shells on."""
    combos, lin, step = [((), (), ())], [0], 1
    for l in ls:
        combos = [tuple(p + (q,) for p, q in zip(c, pw)) for pw in _cart(l) for c in combos]
        lin = [o + step * k for k in range(len(_cart(l))) for o in lin]
        step *= 2 * l + 1

    def at(p):
        v = 0
        for l, q in zip(ls, p):
            v = v * (l + 1) + q
        return v

    dev = w.device
    ix = [torch.tensor([at(c[ax]) for c in combos], device=dev) for ax in range(3)]
    out = torch.zeros((math.prod(len(_cart(l)) for l in ls), n), dtype=torch.float64, device=dev)
    if w.requires_grad or E.requires_grad:
        vals = torch.einsum("cnp,np->cn", E[ix[0], 0] * E[ix[1], 1] * E[ix[2], 2], w)
    else:
        chunk = max(1, int(2e7 // max(1, n * w.shape[1])))
        vals = torch.cat([torch.einsum("cnp,np->cn", E[x, 0] * E[y, 1] * E[zz, 2], w)
                          for x, y, zz in zip(*(i.split(chunk) for i in ix))])
    return out.index_add(0, torch.tensor(lin, device=dev), vals)


def _pair_64(la, lb, za, ca, zb, cb, AB):
    """Block of one shell pair for n geometries AB = A - B (n, 3): (NA NB, n)."""
    n = AB.shape[0]
    a, b = (t.reshape(-1) for t in torch.meshgrid(za, zb, indexing="ij"))
    w = (ca[:, None] * cb[None, :]).reshape(-1)
    p = a + b
    R2 = (AB * AB).sum(1)
    w = w * (math.pi / p) ** 1.5 * torch.exp(-(a * b / p) * R2[:, None])
    X = AB.t()[:, :, None]
    E = _grow({(0, 0): torch.ones((3, n, a.numel()), dtype=torch.float64, device=AB.device)}, (la, lb),
              (-(b / p) * X, (a / p) * X), 0.5 / p)
    return _block_64((la, lb), E, w, n)


def _offsets(ls):
    return np.concatenate([[0], np.cumsum((np.asarray(ls) + 1) * (np.asarray(ls) + 2) // 2)])


def _overlap2c_64(ls, z, coef, A, Bp, sA, sB, dense=False, groups=None):
    """(B, N, N) overlaps, [b, j, i]; `groups` gets each species pair's part instead, as
    (elements, block matrix) (for gradients: `dense` keeps zero coefficients)."""
    off, NZ = _offsets(ls), z.shape[2]
    N, B = int(off[-1]), A.shape[0]
    AB = A.double() - Bp.double()
    out = None if groups is not None else torch.zeros((B, N, N), dtype=torch.float64, device=A.device)
    key = (sA - 1) * NZ + (sB - 1)
    for g in range(NZ * NZ):
        e = torch.nonzero(key == g).flatten()
        if not e.numel():
            continue
        ga, gb = g // NZ, g % NZ
        cols = []
        for t, lb in enumerate(ls):
            rows = []
            for s, la in enumerate(ls):
                ka = torch.arange(z.shape[1], device=A.device) if dense else torch.nonzero(coef[s, :, ga]).flatten()
                kb = torch.arange(z.shape[1], device=A.device) if dense else torch.nonzero(coef[t, :, gb]).flatten()
                na, nb = int(off[s + 1] - off[s]), int(off[t + 1] - off[t])
                if not ka.numel() or not kb.numel():
                    rows.append(torch.zeros((e.numel(), nb, na), dtype=torch.float64, device=A.device))
                    continue
                blk = _pair_64(int(la), int(lb), z[s, ka, ga], coef[s, ka, ga], z[t, kb, gb], coef[t, kb, gb], AB[e])
                rows.append(blk.t().reshape(e.numel(), nb, na))
            cols.append(torch.cat(rows, dim=2))
        S = torch.cat(cols, dim=1)
        if groups is not None:
            groups(e, S)
        else:
            out[e] = S
    return out


def _overlap3c_64(ls, z, coef, X, S):
    """(B, N, N, N) three-center overlaps, [b, k, j, i]; z, coef (ns, K, NZ)."""
    off, NZ = _offsets(ls), z.shape[2]
    N, B, dev = int(off[-1]), X[0].shape[0], X[0].device
    out = torch.zeros((B, N, N, N), dtype=torch.float64, device=dev)
    key = ((S[0] - 1) * NZ + (S[1] - 1)) * NZ + (S[2] - 1)
    for g in range(NZ ** 3):
        e = torch.nonzero(key == g).flatten()
        n = e.numel()
        if not n:
            continue
        sp = (g // (NZ * NZ), g // NZ % NZ, g % NZ)
        live = [[torch.nonzero(coef[s, :, q]).flatten() for s in range(len(ls))] for q in sp]
        R = [x[e].double() for x in X]
        AB, AC, BC = ((R[i] - R[j]) for i, j in ((0, 1), (0, 2), (1, 2)))
        for s in np.ndindex(len(ls), len(ls), len(ls)):
            k = [live[c][s[c]] for c in range(3)]
            if not all(i.numel() for i in k):
                continue
            a, b, c = (t.reshape(-1) for t in torch.meshgrid(*(z[s[i], k[i], sp[i]] for i in range(3)), indexing="ij"))
            w = (coef[s[0], k[0], sp[0]][:, None, None] * coef[s[1], k[1], sp[1]][:, None]
                 * coef[s[2], k[2], sp[2]]).reshape(-1)
            q = a + b + c
            arg = sum((u / q) * (d * d).sum(1)[:, None] for u, d in ((a * b, AB), (a * c, AC), (b * c, BC)))
            w = w * (math.pi / q) ** 1.5 * torch.exp(-arg)
            ab, ac, bc = (d.t()[:, :, None] for d in (AB, AC, BC))
            l = [int(ls[i]) for i in s]
            E = _grow({(0, 0, 0): torch.ones((3, n, a.numel()), dtype=torch.float64, device=dev)}, l,
                      (-(b * ab + c * ac) / q, (a * ab - c * bc) / q, (a * ac + b * bc) / q), 0.5 / q)
            blk = _block_64(l, E, w, n)
            o = [slice(int(off[i]), int(off[i + 1])) for i in s]
            m = [int(off[i + 1] - off[i]) for i in s]
            out[e, o[2], o[1], o[0]] = blk.t().reshape(n, m[2], m[1], m[0])
    return out


def _harmonics_64(X, L):
    """Real solid harmonics, L2-normalised on the sphere, index l^2 + l + m: list of (n,)."""
    x, y, zz = X[:, 0], X[:, 1], X[:, 2]
    r2 = x * x + y * y + zz * zz
    C, S = [torch.ones_like(x)], [torch.zeros_like(x)]
    for m in range(L):
        C.append(x * C[m] - y * S[m])
        S.append(x * S[m] + y * C[m])
    Z = [None] * (L + 1) ** 2
    for m in range(L + 1):
        Q = {m: float(math.prod(range(2 * m - 1, 0, -2))) * torch.ones_like(x)}
        for l in range(m + 1, L + 1):
            Q[l] = ((2 * l - 1) * zz * Q[l - 1] - (l + m - 1) * r2 * Q.get(l - 2, torch.zeros_like(x))) / (l - m)
        for l in range(m, L + 1):
            F = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m == 0:
                Z[l * l + l] = F * Q[l]
            else:
                Z[l * l + l + m] = math.sqrt(2.0) * F * Q[l] * C[m]
                Z[l * l + l - m] = math.sqrt(2.0) * F * Q[l] * S[m]
    return Z


def _orbital_64(case, b, X, sidx, z, D, emit):
    """Calls emit(i, phi_i) for every orbital at X (n, 3)."""
    iR, iY, L = _spec(b)
    poly = _poly(case, b)
    r2 = (X * X).sum(1)
    r = r2.sqrt()
    f = r if case["radial"] == "slater" else r2
    Z = _harmonics_64(X, L)
    for k in range(b.nshells):
        zk, Dk = z[k].t()[sidx - 1], D[k].t()[sidx - 1]
        R = (Dk * torch.exp(-zk * f[:, None])).sum(1)
        if poly[k]:
            R = R * r ** poly[k]
        for i in np.flatnonzero(iR == k + 1):
            emit(int(i), R * Z[iY[i] - 1])


def exact(case, seed):
    kind = case["kind"]
    b, FT, z, D = _overlap_inputs(case, seed)
    z64, D64 = (torch.as_tensor(a, device="cuda") for a in (z, D))
    if kind in ("evaluate_ed", "evaluate_step"):
        X, sidx = _points(case, b, seed)
        n, nOrb = case["nX"], len(_spec(b)[0])
        X = X.double().requires_grad_(True)
        P = torch.empty((nOrb, n), dtype=torch.float64, device="cuda")
        if kind == "evaluate_ed":
            dP = torch.empty((nOrb, n, 3), dtype=torch.float64, device="cuda")

            def emit(i, phi):
                P[i] = phi.detach()
                dP[i] = torch.autograd.grad(phi.sum(), X, retain_graph=True)[0]

            _orbital_64(case, b, X, sidx, z64, D64, emit)
            return P, dP
        ct = _cotangent(case, seed, (nOrb, n)).double()
        z64.requires_grad_(True)
        D64.requires_grad_(True)
        loss = []

        def emit(i, phi):
            P[i] = phi.detach()
            loss.append((phi * ct[i]).sum())

        _orbital_64(case, b, X, sidx, z64, D64, emit)
        dX, dz, dD = torch.autograd.grad(sum(loss), (X, z64, D64))
        return P, dX, dz.permute(2, 1, 0).contiguous(), dD.permute(2, 1, 0).contiguous()
    if kind in ("overlap2c_gb", "overlap3c_gb"):
        ls, nprim, coef, alpha = _gb_arrays(b, z, D)
        if FT == torch.float32:
            coef, alpha = (a.astype(np.float32).astype(np.float64) for a in (coef, alpha))
        zp, cp = np.ones((len(ls), nprim.max(), 1)), np.zeros((len(ls), nprim.max(), 1))
        at = 0
        for s, k in enumerate(nprim):
            zp[s, :k, 0], cp[s, :k, 0] = alpha[at:at + k], coef[at:at + k]
            at += k
        zp, cp = torch.as_tensor(zp, device="cuda"), torch.as_tensor(cp, device="cuda")
        X, _ = _triples(case, b, seed)
        one = torch.ones(case["B"], dtype=torch.int64, device="cuda")
        if kind == "overlap2c_gb":
            return _overlap2c_64(ls, zp, cp, X[0], X[1], one, one)
        return _overlap3c_64(ls, zp, cp, X, [one] * 3)
    if kind == "overlap3c":
        X, S = _triples(case, b, seed)
        return _overlap3c_64(b.ls, z64, _coef_64(b.ls, z64, D64), X, S)
    A, Bp, sA, sB = _pairs(case, b, seed)
    if kind in ("overlap2c", "overlap2c_api"):
        return _overlap2c_64(b.ls, z64, _coef_64(b.ls, z64, D64), A, Bp, sA, sB)
    N, B = b.nbf_total, case["B"]
    if kind == "position":
        ct = _cotangent(case, seed, (B, N, N)).double()
        A = A.double().requires_grad_(True)
        dA = torch.zeros_like(A)

        def back(e, S):
            dA.add_(torch.autograd.grad((S * ct[e]).sum(), A, retain_graph=True)[0])

        _overlap2c_64(b.ls, z64, _coef_64(b.ls, z64, D64), A, Bp, sA, sB, groups=back)
        return dA, -dA
    ct = (_target(case, seed, b, z, D, (A, Bp, sA, sB)) if case["loss"] == "residual"
          else _cotangent(case, seed, (B, N, N))).double()
    z64.requires_grad_(True)
    D64.requires_grad_(True)
    coef = _coef_64(b.ls, z64, D64)
    zc, cc = z64.detach().requires_grad_(True), coef.detach().requires_grad_(True)
    out = torch.empty((B, N, N), dtype=torch.float64, device="cuda")
    dzc, dcc = torch.zeros_like(zc), torch.zeros_like(cc)

    def back(e, S):
        out[e] = S.detach()
        g = 2.0 * (S.detach() - ct[e]) if case["loss"] == "residual" else ct[e]
        gz, gc = torch.autograd.grad((S * g).sum(), (zc, cc))
        dzc.add_(gz)
        dcc.add_(gc)

    _overlap2c_64(b.ls, zc, cc, A, Bp, sA, sB, dense=True, groups=back)
    present = (D64.detach() != 0).any(dim=1, keepdim=True)  # an absent shell has no gradient
    dz, dD = torch.autograd.grad(coef, (z64, D64), dcc)
    return (out, *((t * present).permute(2, 1, 0).contiguous() for t in (dz + dzc, dD)))
