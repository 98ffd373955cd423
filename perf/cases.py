"""Performance cases of the library: what programs built on it run, over the
range of sizes they run it at.

Each case is a dict with an ``op`` (an entry point or the few a program calls
together), its sizes and options:

  solve   Context.cc_solve: the whole CCSD / DCSD iteration from the MP2 guess
  driver  driver.ccdriver "ccsd(t)": the whole call on given integrals
  step    cc_load + cc_step + cc_store: one iteration for a caller that keeps
          the loop (and the amplitudes) on the host
  lambda  Context.lambda_residual: the left-hand equations, the reverse
          direction of the residual
  pert_t  Context.pert_t: the (T) correction of given amplitudes
  dump    df_factors + DFFactors.fock + DFFactors.mo: three-centre integrals,
          a Fock build and the transformation to molecular orbitals

Coupled-cluster cases use seeded factors B[p,q,Q] with a molecule-like decay
whose Hartree-Fock reference is canonical, MP2 doubles and small singles; the
integral cases real molecules (water clusters, alkanes) in their basis sets.
``exact`` gives the results in 64 bits with torch alone.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "elemco.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ecgpu  # noqa: E402
from ecgpu import basis as basis_sets  # noqa: E402
from ecgpu import driver, molecules  # noqa: E402
from ecgpu._lib import ECG_INT_KINETIC, ECG_INT_NUCLEAR, ECG_INT_OVERLAP  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


# ---------------------------------------------------------------- the cases


def _cc(name, op, no, nv, nq, method="ccsd", precision="fp64"):
    return {"name": name, "op": op, "no": no, "nv": nv, "nq": nq, "method": method,
            "precision": precision}


def listed():
    return [
        # a water molecule, cc-pVDZ: the calculation everybody starts with and
        # that scans and test suites repeat; its kernels are tiny
        _cc("solve_water_vdz", "solve", 5, 19, 84),
        # a water dimer (interaction energies), the whole CCSD(T) call
        _cc("driver_water2_vdz", "driver", 8, 38, 168),
        # a water trimer, odd virtual count, one iteration
        _cc("step_water3_vdz", "step", 12, 57, 252),
        # octane: a medium organic molecule, distinguishable-cluster doubles
        _cc("step_octane_vdz_dcsd", "step", 25, 169, 700, method="dcsd"),
        # the water hexamer in cc-pVTZ, the largest single-GPU configuration,
        # in either precision
        _cc("step_water6_vtz", "step", 24, 318, 846),
        _cc("step_water6_vtz_mixed", "step", 24, 318, 846, precision="mixed"),
        # the Lambda equations (gradients, densities) of a water tetramer
        _cc("lambda_water4_vdz", "lambda", 16, 76, 336),
        # (T): a water tetramer; decane in mixed precision (all its triplets);
        # the hexamer's virtual space in FP64 (a small occupied space keeps it
        # to a fraction of a second)
        _cc("pert_t_water4_vdz", "pert_t", 16, 76, 336),
        _cc("pert_t_decane_vdz_mixed", "pert_t", 31, 209, 868, precision="mixed"),
        _cc("pert_t_v318", "pert_t", 6, 318, 846),
        # integrals, Fock build and transformation: a water molecule, and a
        # water tetramer in triple zeta
        {"name": "dump_water_vdz", "op": "dump", "molecule": "water", "size": 1, "zeta": "d",
         "frozen": True},
        {"name": "dump_water4_vtz", "op": "dump", "molecule": "water", "size": 4, "zeta": "t",
         "frozen": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["solve", "driver", "step", "step", "step", "lambda", "pert_t", "pert_t",
                     "dump"])
    if op == "dump":
        mol = rng.choice(["water", "water", "alkane"])
        zeta = rng.choice(["d", "t"]) if mol == "water" else "d"
        lo, hi = (1, 8) if mol == "alkane" else (1, 3) if zeta == "t" else (2, 6)
        return {"op": op, "molecule": mol, "size": rng.randint(lo, hi), "zeta": zeta,
                "frozen": rng.random() < 0.5}
    small = op in ("solve", "driver")
    no = _log(rng, 4, 10 if small else 16 if op == "lambda" else 25)
    hi = 60 if small else 100 if op == "lambda" else 200
    nv = max(_log(rng, 15, hi), no + 2)
    return {"op": op, "no": no, "nv": nv, "nq": int((no + nv) * rng.uniform(2.5, 3.6)),
            "method": "ccsd" if op in ("driver", "pert_t") else rng.choice(["ccsd", "dcsd"]),
            "precision": "fp64" if op == "lambda" or rng.random() < 0.6 else "mixed"}


# ---------------------------------------------------------------- inputs


def _perm2(T):
    """T[b,a,j,i] of T[a,b,i,j] (torch order [j,i,b,a] of the F-ordered array)."""
    return T.permute(1, 0, 3, 2)


def _system(case, seed):
    """Factors B[Q,q,p], h, orbital energies and amplitudes T1[i,a], T2[j,i,b,a]
    on the GPU; C-ordered here, so F-ordered with reversed indices in numpy."""
    no, nv, nq = case["no"], case["nv"], case["nq"]
    n = no + nv
    g = torch.Generator(device=DEV).manual_seed(1000003 * (seed % 100003) + 17)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=F64)  # noqa: E731
    uni = lambda k, lo, hi: lo + (hi - lo) * torch.rand(  # noqa: E731
        k, generator=g, device=DEV, dtype=F64)
    eo = uni(no, -1.4, -0.4).sort().values
    ev = uni(nv, 0.1, 4.0).sort().values
    B = rnd(nq, n, n)
    for q in range(0, nq, 64):
        B[q:q + 64] += B[q:q + 64].transpose(1, 2).clone()
    w = 10.0 ** (-6.0 * torch.arange(nq, device=DEV, dtype=F64) / max(nq - 1, 1))
    B *= (w / math.sqrt(2.0 * n))[:, None, None]
    ov = B[:, :no, no:].reshape(nq, no * nv)
    D = eo[:, None] - ev[None, :]
    D = (D.reshape(-1, 1) + D.reshape(1, -1)).view(no, nv, no, nv)
    K = (ov.T @ ov).view(no, nv, no, nv)
    emp2 = float((K * (2.0 * K - K.transpose(1, 3)) / D).sum())
    s = (-0.05 * no / emp2) ** 0.25  # MP2 correlation of -0.05 Eh an orbital
    B *= s
    T2 = (K * s ** 2 / D).permute(2, 0, 3, 1).contiguous()  # [j,i,b,a]
    T1 = 0.02 * rnd(no, nv) / (ev[None, :] - eo[:, None] + 1.0)
    J = B[:, :no, :no].diagonal(dim1=1, dim2=2).sum(1)
    X = B[:, :, :no].reshape(nq, n, no)
    h = torch.diag(torch.cat([eo, ev])) - 2.0 * torch.einsum("Qpq,Q->pq", B, J)
    h += torch.einsum("Qpk,Qqk->pq", X, X)
    return B, h, eo, ev, T1, T2


def _multipliers(T1, T2):
    """Multipliers of the size a left-hand iteration starts from: U2 = 2T2 - T2^x."""
    return 2.0 * T1, (2.0 * T2 - T2.transpose(0, 1)).contiguous()


def _host(x, pinned=False):
    """numpy F-ordered view of the host copy of a C-ordered tensor."""
    h = torch.empty(x.shape, dtype=x.dtype, pin_memory=pinned and x.is_cuda)
    h.copy_(x)
    return h.numpy().T


def _molecule(case, seed):
    n = case["size"]
    if case["molecule"] == "water":
        if n > 1:
            return molecules.water_cluster(n, seed=seed)
        xyz = molecules.WATER_XYZ * (1.0 + 0.02 * np.random.default_rng(seed).random())
        return molecules.Molecule(["O", "H", "H"], xyz)
    return molecules.alkane(n, seed=seed)


def _shells(case, seed):
    mol = _molecule(case, seed)
    z = case["zeta"]
    ao, fit = (basis_sets.shells(basis_sets.load(f"cc-pv{z}z{s}"), mol.symbols, mol.xyz)
               for s in ("", "-mpfit"))
    return mol, ao, fit


def _core(case, mol):
    return mol.ncore() if case["frozen"] else 0


def _dump_inputs(ctx, case, seed):
    """Basis shells, fitting matrix M (M M^T = (P|Q)^-1), h and S-orthonormal orbitals."""
    mol, ao, fit = _shells(case, seed)
    M = np.asfortranarray(np.linalg.inv(np.linalg.cholesky(ctx.int2c2e(fit))).T)
    h = np.asfortranarray(ctx.int1e(ECG_INT_KINETIC, ao)
                          + ctx.int1e(ECG_INT_NUCLEAR, ao, mol.charges, mol.xyz))
    s, U = np.linalg.eigh(ctx.int1e(ECG_INT_OVERLAP, ao))
    X = (U / np.sqrt(s)) @ U.T
    _, V = np.linalg.eigh(X @ h @ X)
    return mol, ao, fit, M, h, np.asfortranarray(X @ V)


def prepare(case, seed):
    EC = driver.ECInfo(scr=tempfile.gettempdir())
    ctx = EC.context()  # loads the packaged GEMM table, as ccdriver does
    op = case["op"]
    st = {"case": case, "EC": EC, "ctx": ctx}
    if op == "dump":
        mol, ao, fit, M, h, C = _dump_inputs(ctx, case, seed)
        st.update(ao=ao, fit=fit, M=M, h=h, nocc=mol.nelec // 2,
                  occ=np.asfortranarray(C[:, :mol.nelec // 2]),
                  act=np.asfortranarray(C[:, _core(case, mol):]))
        return st
    B, h, eo, ev, T1, T2 = _system(case, seed)
    if op in ("solve", "driver"):  # these start from MP2
        T1 = torch.zeros_like(T1)
    Bh, hh = _host(B), _host(h)
    st["T"] = [_host(T1, True), _host(T2, True)]
    if op == "lambda":
        st["U"] = [_host(x) for x in _multipliers(T1, T2)]
    if op == "step":
        st["out"] = [_host(torch.zeros_like(T1), True), _host(torch.zeros_like(T2), True)]
    del B, h, T1, T2
    if op == "driver":
        EC.fd = driver.FDump(hh, 0.0, 2 * case["no"], B=Bh)
        EC.set("cc", save="")
        EC.set("gpu", precision=case["precision"])
        return st
    ctx.set_precision(ecgpu.ECG_PREC_MIXED if case["precision"] == "mixed"
                      else ecgpu.ECG_PREC_FP64)
    ctx.set_system(Bh, hh, 0.0, case["no"])
    return st


# ---------------------------------------------------------------- one pass


def run(st):
    case, ctx = st["case"], st["ctx"]
    op, dc = case["op"], case.get("method") == "dcsd"
    if op == "dump":
        with ctx.df_factors(st["ao"], st["fit"], st["M"]) as AAL:
            return {"F": AAL.fock(st["h"], st["occ"]), "B": AAL.mo(st["act"])}
    if op == "driver":
        out = driver.ccdriver(st["EC"], "ccsd(t)")
        E = np.array([out[k] for k in ("HF", "MP2c", "CCSDc", "CCSD", "[T]", "(T)", "CCSD(T)")])
        return {"E": E, "T": ctx.cc_store(), "iterations": out["iterations"]}
    T1, T2 = st["T"]
    if op == "solve":
        r = ctx.cc_solve(T1, T2, dc=dc)
        return {"E": r["E"], "T1": r["T1"], "T2": r["T2"], "iterations": r["iterations"]}
    if op == "step":
        ctx.cc_load(T1, T2)
        e = ctx.cc_step(dc=dc)
        return {"E": e[:3].copy(), "T": ctx.cc_store(*st["out"])}
    if op == "lambda":
        return ctx.lambda_residual(T1, T2, *st["U"], dc=dc)
    return np.array(ctx.pert_t(T1, T2))


# ---------------------------------------------------------------- work


def _triplets(no):
    for k in range(no):
        for j in range(k + 1):
            for i in range(j + 1):
                if not (i == j == k):
                    yield i, j, k, 1.0 if i == j or j == k else 2.0


def work(case):
    """What a pass cannot do without: the ladder over a<=b, c<=d, i<=j and its
    integrals (ac|bd) over a<=b, the o^3 v^3 and o^4 v^2 products; (T): the
    twelve v^4 and o v^3 products a triplet; inputs and outputs once."""
    if case["op"] == "dump":
        mol, ao, fit = _shells(case, 1)
        n, m, no = ao.nbf, fit.nbf, mol.nelec // 2
        na = n - _core(case, mol)
        return {"bytes": 8.0 * (m * m + 3 * n * n + na * na * m),
                "flops": n * n * float(m) * m + 3.0 * no * n * n * m + 2.0 * na * n * n * m
                + na * na * n * float(m)}
    o, v, Q = float(case["no"]), float(case["nv"]), float(case["nq"])
    rings = (8.0 if case["method"] == "dcsd" else 16.0) * o ** 3 * v ** 3
    it = o * o * v ** 4 / 2 + Q * v ** 4 + rings + 4 * o ** 4 * v ** 2
    nt = sum(1 for _ in _triplets(case["no"]))
    pt = nt * (12 * v ** 4 + 12 * o * v ** 3) + 2 * Q * o * v ** 3
    b = 8.0 * ((o + v) ** 2 * Q + o * o * v * v)
    t2 = 8.0 * o * o * v * v
    return {"solve": {"bytes": b + t2, "flops": 10 * it},
            "driver": {"bytes": b, "flops": 10 * it + pt},
            "step": {"bytes": b + t2, "flops": it},
            "lambda": {"bytes": b + 2 * t2, "flops": it + rings + 2 * Q * o * v ** 3},
            "pert_t": {"bytes": b, "flops": pt}}[case["op"]]


def tolerance(case):
    # about four times the error against ``exact``: mixed precision 1e-5 (T1 of a
    # CCSD step) and 3e-6 ((T)); FP64 1e-14, which the fitting metric's inverse
    # amplifies to 4e-12 in the factors and DIIS to 4e-11 in a solve's iterates
    if case.get("precision") == "mixed":
        return {"rel": 4e-5, "max": 5e-3}
    if case["op"] in ("solve", "driver"):
        return {"rel": 2e-10, "max": 1e-8}
    return {"rel": 1e-10 if case["op"] == "dump" else 1e-12}


# ---------------------------------------------------------------- 64-bit results


def _dressed(B, h, T1):
    """T1-dressed factors (oo, vo, ov, vv) and Fock matrix (all [p,q], rows first)."""
    no = T1.shape[0]
    t = T1.T  # [a,i]
    n = h.shape[0]
    X = torch.zeros(n, n, dtype=F64, device=B.device)
    X[no:, :no] = t
    one = torch.eye(n, dtype=F64, device=B.device)
    L, R = one - X, one + X
    dB = L @ B @ R
    dh = L @ h @ R
    J = dB[:, :no, :no].diagonal(dim1=1, dim2=2).sum(1)
    f = dh + 2.0 * torch.einsum("Qpq,Q->pq", dB, J)
    f = f - torch.einsum("Qpk,Qkq->pq", dB[:, :, :no], dB[:, :no, :])
    return dB, f


def _residual(B, h, T1, T2, dc):
    """Closed-shell CCSD / DCSD residuals in the layouts of T1[i,a], T2[j,i,b,a]."""
    no = T1.shape[0]
    o, v = slice(0, no), slice(no, None)
    dB, f = _dressed(B, h, T1)
    es = torch.einsum
    t = T2.permute(3, 2, 1, 0)  # [a,b,i,j]
    tt = 2.0 * t - t.transpose(0, 1)
    bov = B[:, o, v]
    oo, vo, vv = dB[:, o, o], dB[:, v, o], dB[:, v, v]
    g = es("Qkc,Qld->klcd", bov, bov)
    # singles
    W = es("cdil,Qld->Qci", tt, bov)
    R1 = f[v, o] + es("Qac,Qci->ai", vv, W) - es("Qaj,Qji->ai", W, oo)
    R1 = R1 + es("abij,jb->ai", tt, f[o, v])
    # doubles: particle ladder one a at a time, hole ladder
    nv = t.shape[0]
    tm = t.reshape(nv * nv, no * no)
    rows = []
    for a in range(nv):
        Va = es("Qc,Qbd->bcd", vv[:, a], vv).reshape(nv, nv * nv)
        rows.append((Va @ tm).view(nv, no, no))
    R2 = torch.stack(rows)
    I = es("Qki,Qlj->klij", oo, oo)
    if not dc:
        I = I + es("klcd,cdij->klij", g, t)
    R2 = R2 + es("abkl,klij->abij", t, I) + es("Qai,Qbj->abij", vo, vo)
    if not dc:
        R2 = R2 + es("lcaj,cbil->abij", es("klcd,adkj->lcaj", g, t), t)
    fac = 0.5 if dc else 1.0
    xv = f[v, v] - fac * es("klcd,cakl->ad", g, tt)
    xo = f[o, o] + fac * es("klcd,cdil->ki", g, tt)
    P = es("ad,dbij->abij", xv, t) - es("ki,abkj->abij", xo, t)
    W = es("Qai,Qkc->akic", vo, bov) + 0.5 * es("klcd,adil->akic", g, tt)
    P = P + es("akic,cbkj->abij", W, tt)
    if not dc:
        P = P - es("lcai,cblj->abij", es("klcd,daki->lcai", g, t), tt - t)
    W = es("Qac,Qki->akci", vv, oo)
    P = P - es("akci,cbkj->abij", W, t) - es("bkci,ackj->abij", W, t)
    R2 = R2 + P + P.permute(1, 0, 3, 2)
    return R1.T, R2.permute(3, 2, 1, 0)


def _energies(B, h, T1, T2):
    """(same-spin, opposite-spin) correlation energies of amplitudes, and 2 f.T1."""
    no = T1.shape[0]
    g = torch.einsum("Qia,Qjb->jiba", B[:, :no, no:], B[:, :no, no:])
    f = _dressed(B, h, torch.zeros_like(T1))[1]
    tau = T2 + torch.einsum("ia,jb->jiba", T1, T1)
    d, x = (tau * g).sum(), (tau * g.transpose(2, 3)).sum()
    return d - x, d, 2.0 * (f[:no, no:] * T1).sum()


def _cs_dot(X, Y):
    """Closed-shell dot product of (singles, doubles) vectors."""
    return float(2.0 * (X[0] * Y[0]).sum() + 2.0 * (X[1] * Y[1]).sum()
                 - (X[1] * Y[1].transpose(2, 3)).sum())


def _iterate(case, B, h, eo, ev, T1, T2, steps=None):
    """Iterations with level shifts 0.15 / 0.2 and DIIS over six vectors;
    `steps` of them, or until the default thresholds are met."""
    dc = case["method"] == "dcsd"
    D1 = ev[None, :] - eo[:, None]
    D2 = (D1[:, None, :, None] + D1[None, :, None, :]).contiguous()
    amps, res, Bm, nxt = [None] * 6, [None] * 6, np.zeros((6, 6)), 0
    nd = 0
    for it in range(1, (steps or 50) + 1):
        R1, R2 = _residual(B, h, T1, T2, dc)
        ss, os_, f1 = (float(x) for x in _energies(B, h, T1, T2))
        no = T1.shape[0]
        g = (T2 * R2).sum(), (T2 * R2.transpose(2, 3)).sum()
        r1 = 2.0 * float((R1 * T1).sum())
        E = (ss + os_ + f1 + float(2.0 * g[0] - g[1]) + r1, ss + float(g[0] - g[1]),
             os_ + float(g[0]))
        norm = _cs_dot((R1, R2), (R1, R2))
        T1, T2 = T1 - R1 / (D1 + 0.15), T2 - R2 / (D2 + 0.2)
        nd = min(nd + 1, 6)
        cur = nxt
        amps[cur], res[cur] = (T1, T2), (R1, R2)
        for i in range(nd):
            Bm[i, cur] = Bm[cur, i] = _cs_dot((R1, R2), res[i])
        A = -np.ones((nd + 1, nd + 1))
        A[:nd, :nd] = Bm[:nd, :nd]
        A[nd, nd] = 0.0
        c = np.linalg.pinv(A, rcond=2.2e-16)[:, nd] * -1.0
        if nd == 1 and cur == 0 and Bm[0, 0] > 10.0:
            nd = 0
        else:
            nxt = nd if nd < 6 else min((i for i in range(nd) if i != cur),
                                        key=lambda i: abs(c[i]))
            T1 = sum(c[i] * amps[i][0] for i in range(nd))
            T2 = sum(c[i] * amps[i][1] for i in range(nd))
        if steps is None:
            ss, os_, f1 = (float(x) for x in _energies(B, h, T1, T2))
            if norm < 1e-10 and abs(ss + os_ + f1 - E[0]) < 1e-6:
                break
    return E, T1, T2


def _pert_t(B, h, eo, ev, T1, T2):
    """(T) and [T] from K = P[W] over occupied triplets."""
    no, nv = T1.shape
    o, v = slice(0, no), slice(no, None)
    es = torch.einsum
    t = T2.permute(3, 2, 1, 0).contiguous()
    g = es("Qia,Qjb->abij", B[:, o, v], B[:, o, v])
    f = _dressed(B, h, torch.zeros_like(T1))[1]
    ovoo = es("Qlj,Qck->ljck", B[:, o, o], B[:, v, o])
    bvv = B[:, v, v].reshape(B.shape[0], -1)
    vvvo = [(B[:, v, k].T @ bvv).view(nv, nv, nv) for k in range(no)]  # [c,b,d]
    D3 = ev[:, None, None] + ev[None, :, None] + ev[None, None, :]

    def W(x, y, z):
        w = (t[:, :, x, y] @ vvvo[z].reshape(nv * nv, nv).T).view(nv, nv, nv).transpose(1, 2)
        return w - es("abl,lc->abc", t[:, :, x, :], ovoo[:, y, :, z])

    et = eb = 0.0
    for i, j, k, fac in _triplets(no):
        K = W(i, j, k) + W(j, i, k).transpose(0, 1) + W(i, k, j).transpose(1, 2)
        K = K + W(k, j, i).permute(2, 1, 0) + W(j, k, i).permute(2, 0, 1)
        K = K + W(k, i, j).permute(1, 2, 0)
        X = 4 * K - 2 * (K.permute(0, 2, 1) + K.permute(2, 1, 0) + K.permute(1, 0, 2))
        X = (X + K.permute(2, 0, 1) + K.permute(1, 2, 0)) / (eo[i] + eo[j] + eo[k] - D3)
        eb += fac * float((K * X).sum())
        for p, q, r, ax in ((i, j, k, "abc,bc->a"), (j, i, k, "abc,ac->b"), (k, i, j, "abc,ab->c")):
            et += fac * float((es(ax, X, g[:, :, q, r]) * T1[p]).sum()
                              + (es(ax, X, t[:, :, q, r]) * f[p, v]).sum())
    return et + eb, eb


def _lambda(case, B, h, T1, T2, U1, U2):
    """Gradient of E + <U|R> with respect to the amplitudes."""
    T1, T2 = T1.clone().requires_grad_(), T2.clone().requires_grad_()
    R1, R2 = _residual(B, h, T1, T2, case["method"] == "dcsd")
    L = sum(_energies(B, h, T1, T2)) + (U1 * R1).sum() + (U2 * R2).sum()
    G1, G2 = torch.autograd.grad(L, (T1, T2))
    return G1, 0.5 * (G2 + _perm2(G2))


# -- Gaussian integrals (McMurchie and Davidson 1978), batched over primitives


def _cartesians(l):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


def _solid(l):
    """Real solid harmonics m = -l..l in Cartesian monomials (unnormalised)."""
    idx = {c: n for n, c in enumerate(_cartesians(l))}
    out = np.zeros((2 * l + 1, len(idx)))
    for m in range(-l, l + 1):
        am, odd = abs(m), 1 if m < 0 else 0
        for t in range((l - am) // 2 + 1):
            for u in range(t + 1):
                for k in range(odd, am + 1, 2):
                    c = (-1) ** (t + (k - odd) // 2) * 0.25 ** t * math.comb(l, t)
                    c *= math.comb(l - t, am + t) * math.comb(t, u) * math.comb(am, k)
                    out[m + l, idx[(2 * t + am - 2 * u - k, 2 * u + k, l - 2 * t - am)]] += c
    return torch.tensor(out, dtype=F64, device=DEV)


def _hermite(la, lb, p, pa, pb):
    """E[i][j][t] of the 1-D product over a batch of primitive pairs."""
    E = [[None] * (lb + 1) for _ in range(la + 1)]
    zero, h = torch.zeros_like(p), 0.5 / p

    def up(e, x):
        n = len(e)
        return [x * (e[t] if t < n else zero) + (h * e[t - 1] if t else zero)
                + ((t + 1) * e[t + 1] if t + 1 < n else zero) for t in range(n + 1)]

    for i in range(la + 1):
        E[i][0] = [torch.ones_like(p)] if i == 0 else up(E[i - 1][0], pa)
        for j in range(1, lb + 1):
            E[i][j] = up(E[i][j - 1], pb)
    return E


def _boys(m, T):
    """F_0..F_m by the incomplete gamma function and downward recursion."""
    a = torch.full_like(T, m + 0.5)
    Ts = T.clamp(min=1e-13)
    top = 0.5 * math.gamma(m + 0.5) * torch.special.gammainc(a, Ts) * Ts ** -(m + 0.5)
    top = torch.where(T < 1e-2, sum((-T) ** k / (math.factorial(k) * (2 * m + 2 * k + 1))
                                    for k in range(8)), top)
    F, et = [top], torch.exp(-T)
    for n in range(m, 0, -1):
        F.insert(0, (2 * T * F[0] + et) / (2 * n - 1))
    return F


def _coulomb_tensor(L, alpha, X):
    """R_tuv, t+u+v <= L, as a dict, for distances X = (x, y, z)."""
    F = _boys(L, alpha * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2))
    R = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2 * alpha) ** n * F[n]}
        for s in range(1, L - n + 1):
            for t, u, w in _cartesians(s):
                d = 0 if t else 1 if u else 2
                k = [t, u, w]
                k[d] -= 1
                r = X[d] * R[tuple(k)]
                if k[d]:
                    c = k[d]
                    k[d] -= 1
                    r = r + c * R[tuple(k)]
                new[(t, u, w)] = r
        R = new
    return R


class _Prims:
    """Shells of one basis as flat primitives grouped by angular momentum."""

    def __init__(self, sh):
        self.sh, off, c0 = sh, 0, 0
        self.rows = {}  # l -> [shell, function offset, primitive slice, centre]
        for s, l in enumerate(sh.l):
            k = int(sh.nprim[s])
            self.rows.setdefault(int(l), []).append((c0, slice(off, off + k),
                                                     sh.centre[3 * s:3 * s + 3]))
            off, c0 = off + k, c0 + 2 * int(l) + 1
        self.n = c0

    def block(self, l):
        """(exponent, coefficient, xyz, shell index) of all primitives of degree l,
        contracted functions scaled to unit norm."""
        e, c, x, idx = [], [], [], []
        for k, (_, sl, xyz) in enumerate(self.rows[l]):
            a = self.sh.exps[sl]
            d = self.sh.coefs[sl] * a ** ((2 * l + 3) / 4.0)
            p = a[:, None] + a[None, :]
            # <r^l|r^l> of one solid harmonic, the angular part left to _scale
            d = d / math.sqrt(float((d[:, None] * d[None, :] / p ** (l + 1.5)).sum()))
            e.append(a), c.append(d), idx.append(np.full(len(a), k))
            x.append(np.repeat(xyz[None, :], len(a), 0))
        f = lambda z: torch.tensor(np.concatenate(z), device=DEV)  # noqa: E731
        return f(e), f(c), f(x), f(idx)

    def offsets(self, l):
        return [r[0] for r in self.rows[l]]


def _scale(l):
    """Solid harmonics scaled so that the radially normalised shell has unit norm."""
    S = _solid(l)
    dfact = lambda k: math.prod(range(k, 0, -2)) if k > 0 else 1  # noqa: E731
    C = _cartesians(l)
    G = torch.zeros(len(C), len(C), dtype=F64, device=DEV)
    for i, a in enumerate(C):
        for j, b in enumerate(C):
            s = [x + y for x, y in zip(a, b)]
            if not any(k % 2 for k in s):
                G[i, j] = math.pi ** 1.5 * math.prod(dfact(k - 1) / 2.0 ** (k // 2) for k in s)
    return S / (S @ G @ S.T).diagonal().sqrt()[:, None]


def _three_centre(ao, fit):
    """(mn|P) as [P, n, m]."""
    A, P = _Prims(ao), _Prims(fit)
    out = torch.zeros(P.n, A.n, A.n, dtype=F64, device=DEV)
    for la in A.rows:
        ea, ca, xa, ia = A.block(la)
        for lb in A.rows:
            if lb > la:
                continue
            eb, cb, xb, ib = A.block(lb)
            na, nb = len(A.rows[la]), len(A.rows[lb])
            pi, pj = (z.reshape(-1) for z in torch.meshgrid(
                torch.arange(len(ea), device=DEV), torch.arange(len(eb), device=DEV),
                indexing="ij"))
            p = ea[pi] + eb[pj]
            ctr = (ea[pi, None] * xa[pi] + eb[pj, None] * xb[pj]) / p[:, None]
            k = torch.exp(-ea[pi] * eb[pj] / p * ((xa[pi] - xb[pj]) ** 2).sum(1))
            k = k * ca[pi] * cb[pj]
            pair = ia[pi] * nb + ib[pj]
            keep = k.abs() > 1e-30
            pi, pj, p, ctr, k, pair = (z[keep] for z in (pi, pj, p, ctr, k, pair))
            E = [_hermite(la, lb, p, ctr[:, d] - xa[pi, d], ctr[:, d] - xb[pj, d])
                 for d in range(3)]
            tuvs = [c for s in range(la + lb + 1) for c in _cartesians(s)]
            # Hermite coefficients of the spherical pair: [pair primitive, sa, sb, tuv]
            H = torch.zeros(len(p), len(_cartesians(la)), len(_cartesians(lb)), len(tuvs),
                            dtype=F64, device=DEV)
            for x, a in enumerate(_cartesians(la)):
                for y, b in enumerate(_cartesians(lb)):
                    for z, tuv in enumerate(tuvs):
                        if all(tuv[d] <= a[d] + b[d] for d in range(3)):
                            H[:, x, y, z] = math.prod(
                                E[d][a[d]][b[d]][tuv[d]] for d in range(3)) * k
            H = torch.einsum("pxyz,sx,ty->pstz", H, _scale(la), _scale(lb))
            for lc in P.rows:
                ec, cc, xc, ic = P.block(lc)
                q = ec
                Ec = _hermite(lc, 0, q, torch.zeros_like(q), torch.zeros_like(q))
                carts = _cartesians(lc)
                ks = [c for s in range(lc + 1) for c in _cartesians(s)]
                Hc = torch.zeros(len(q), len(carts), len(ks), dtype=F64, device=DEV)
                for x, a in enumerate(carts):
                    for z, tuv in enumerate(ks):
                        if all(tuv[d] <= a[d] for d in range(3)):
                            e = math.prod(Ec[a[d]][0][tuv[d]] for d in range(3))
                            Hc[:, x, z] = e * cc * (-1) ** sum(tuv)
                Hc = torch.einsum("qxz,sx->qsz", Hc, _scale(lc))
                nc, L = len(P.rows[lc]), la + lb + lc
                acc = torch.zeros(na * nb, nc, 2 * la + 1, 2 * lb + 1, 2 * lc + 1, dtype=F64,
                                  device=DEV)
                step = max(1, 20_000_000 // (len(q) * max(len(tuvs) * len(ks), L ** 3 + 1)))
                for s in range(0, len(p), step):
                    sl = slice(s, s + step)
                    pp, qq = p[sl, None], q[None, :]
                    R = _coulomb_tensor(L, pp * qq / (pp + qq),
                                        [ctr[sl, None, d] - xc[None, :, d] for d in range(3)])
                    pref = 2 * math.pi ** 2.5 / (pp * qq * (pp + qq).sqrt())
                    Rm = torch.stack([torch.stack([R[tuple(x + y for x, y in zip(u, w))]
                                                   for w in ks]) for u in tuvs])
                    V = torch.einsum("uwpq,qcw->pquc", Rm * pref, Hc)
                    V = torch.einsum("pstu,pquc->pqstc", H[sl], V)
                    Vc = torch.zeros(V.shape[0], nc, *V.shape[2:], dtype=F64, device=DEV)
                    Vc.index_add_(1, ic, V)
                    acc.index_add_(0, pair[sl], Vc)
                acc = acc.view(na, nb, nc, 2 * la + 1, 2 * lb + 1, 2 * lc + 1)
                ix = lambda offs, l: (torch.tensor(offs)[:, None]  # noqa: E731
                                      + torch.arange(2 * l + 1)).reshape(-1).to(DEV)
                blk = acc.permute(2, 5, 1, 4, 0, 3).reshape(
                    nc * (2 * lc + 1), nb * (2 * lb + 1), na * (2 * la + 1))
                I, J, K = ix(P.offsets(lc), lc), ix(A.offsets(lb), lb), ix(A.offsets(la), la)
                out[I[:, None, None], J[None, :, None], K[None, None, :]] = blk
                out[I[:, None, None], K[None, :, None], J[None, None, :]] = blk.transpose(1, 2)
    return out


def exact(case, seed):
    op = case["op"]
    if op == "dump":
        with ecgpu.Context(0) as ctx:
            mol, ao, fit, M, h, C = _dump_inputs(ctx, case, seed)
        G = _three_centre(ao, fit)
        t = lambda x: torch.tensor(np.ascontiguousarray(x), device=DEV)  # noqa: E731
        AAL = torch.einsum("Pnm,PL->Lnm", G, t(M))
        occ, act = t(C[:, :mol.nelec // 2]), t(C[:, _core(case, mol):])
        Y = torch.einsum("Lnm,mj->Lnj", AAL, occ)
        F = t(h) + 2.0 * torch.einsum("Lnm,L->nm", AAL, torch.einsum("Lnj,nj->L", Y, occ))
        F = F - torch.einsum("Lmj,Lnj->mn", Y, Y)
        B = act.T @ AAL @ act  # [L,q,p]
        return {"F": F.cpu().numpy(), "B": B.cpu().numpy().T}
    B, h, eo, ev, T1, T2 = _system(case, seed)
    back = lambda x: x.detach().cpu().numpy().T  # noqa: E731
    if op == "lambda":
        return tuple(back(x) for x in _lambda(case, B, h, T1, T2, *_multipliers(T1, T2)))
    if op == "pert_t":
        return np.array(_pert_t(B, h, eo, ev, T1, T2))
    if op == "step":
        E, T1, T2 = _iterate(case, B, h, eo, ev, T1, T2, steps=1)
        return {"E": np.array(E), "T": (back(T1), back(T2))}
    E, T1, T2 = _iterate(case, B, h, eo, ev, torch.zeros_like(T1), T2)
    if op == "solve":
        return {"E": np.float64(E[0]), "T1": back(T1), "T2": back(T2), "iterations": None}
    f = _dressed(B, h, torch.zeros_like(T1))[1].diagonal()
    hf = float((f + h.diagonal())[:case["no"]].sum())
    _, _, _, _, _, M2 = _system(case, seed)
    mp2 = sum(float(x) for x in _energies(B, h, torch.zeros_like(T1), M2)[:2])
    et, eb = _pert_t(B, h, eo, ev, T1, T2)
    return {"E": np.array([hf, mp2, E[0], E[0] + hf, eb, et, E[0] + et + hf]),
            "T": (back(T1), back(T2)), "iterations": None}
