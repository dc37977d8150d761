"""Performance cases of the sigma build, the Davidson solve, the pair-domain all-external operator and the projections.

Each case is a plain dict; prepare() makes what a program holds before the call (operator, context, vectors on the
GPU), run() is one pass through the public entry points, work() the bytes and operations a pass cannot do without
and exact() the same result in 64 bits by plain torch, where the reference is closed-shell and its CSF order is
short to state.

Kinds
  sigma     SigmaBuilder.htimesc_device on a synthetic operator of molecular magnitude (local pair domains when
            dmax > 0)
  chain     the same on the serving stream's requests (an H_n chain's sizes in cc-pVDZ, CAS(2,2) references)
  davidson  SigmaBuilder.davidson on either operator
  pairs     LocalAllExternal.apply_device over pairs with domains of their own
  dots      SigmaBuilder.dots, the projections of a caller-driven Davidson
"""
import math

import numpy as np
import torch

import tigerci_b200 as T
from tigerci_b200 import local as tlocal
from tigerci_b200 import serve


def listed():
    return [
        # the smallest calls: one sigma build at the size of a short H chain (launch-bound), projections on a small vector
        dict(name="sigma_h8_mixed", kind="chain", atoms=8, precision="tf32x3", roots=0),
        dict(name="dots_3x40539", kind="dots", rows=3, length=40539),
        # projections of a new vector on the Davidson subspace of the kernel-scale configuration
        dict(name="dots_27x1971105", kind="dots", rows=27, length=1971105),
        # a whole three-root solve of a mid-sized chain of the serving stream, plain FP64
        dict(name="solve_h12_fp64", kind="chain", atoms=12, precision="fp64", roots=3),
        # an open-shell multireference space with odd sizes (doublet, three references, 101 virtuals)
        dict(name="sigma_doublet_101_fp64", kind="sigma", inactive=5, active=3, act_el=3, mult=2, refs=3, virt=101,
             nchol=403, precision="fp64", roots=0, dmin=0, dmax=0),
        # the kernel-scale configuration (8 inactive + 8 active, 240 virtuals), both forms
        dict(name="sigma_240_fp64", kind="sigma", inactive=8, active=8, act_el=0, mult=1, refs=1, virt=240,
             nchol=800, precision="fp64", roots=0, dmin=0, dmax=0),
        dict(name="sigma_240_mixed", kind="sigma", inactive=8, active=8, act_el=0, mult=1, refs=1, virt=240,
             nchol=800, precision="tf32x3", roots=0, dmin=0, dmax=0),
        # the benchmark's solve: one root of that configuration in the mixed form
        dict(name="solve_240_mixed", kind="sigma", inactive=8, active=8, act_el=0, mult=1, refs=1, virt=240,
             nchol=800, precision="tf32x3", roots=1, dmin=0, dmax=0),
        # many closed-shell pairs: the size of a sigma build of a larger molecule (24 correlated pairs, 173 virtuals)
        dict(name="sigma_24x173_fp64", kind="sigma", inactive=24, active=0, act_el=0, mult=1, refs=1, virt=173,
             nchol=700, precision="fp64", roots=0, dmin=0, dmax=0),
        # the pair-domain all-external operator by itself, FP64 (Cholesky form)
        dict(name="pairs_150_fp64", kind="pairs", pairs=150, n_int=17, virt=300, dmin=20, dmax=150, nchol=900,
             precision="fp64"),
        # local correlation: sigma builds over pair domains, both forms
        dict(name="sigma_local_20x300_fp64", kind="sigma", inactive=20, active=0, act_el=0, mult=1, refs=1, virt=300,
             nchol=600, precision="fp64", roots=0, dmin=20, dmax=160),
        dict(name="sigma_local_20x300_mixed", kind="sigma", inactive=20, active=0, act_el=0, mult=1, refs=1, virt=300,
             nchol=600, precision="tf32x3", roots=0, dmin=20, dmax=160),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "local", "chain", "davidson", "pairs", "dots"])
    prec = rng.choice(["fp64", "tf32x3"])
    if kind == "dots":
        return dict(kind="dots", rows=rng.randint(1, 40), length=_log(rng, 20000, 2000000))
    if kind == "chain":
        return dict(kind="chain", atoms=rng.choice([8, 10, 12, 14, 16, 18]), precision=prec, roots=rng.randint(0, 3))
    if kind == "pairs":
        n = rng.randint(8, 17)
        dmin = rng.randint(10, 40)
        return dict(kind="pairs", pairs=rng.randint(n, min(150, n * (n + 1) // 2)), n_int=n, virt=rng.randint(160, 300),
                    dmin=dmin, dmax=rng.randint(dmin + 20, 150), nchol=rng.randint(300, 900), precision="fp64")
    if kind == "local":
        virt = rng.randint(120, 300)
        dmin = rng.randint(10, 40)
        return dict(kind="sigma", inactive=rng.randint(8, 20), active=0, act_el=0, mult=1, refs=1, virt=virt,
                    nchol=2 * virt, precision=prec, roots=0, dmin=dmin, dmax=min(160, dmin + rng.randint(30, virt // 2)))
    virt = _log(rng, 24, 240)
    c = dict(kind="sigma", virt=virt, nchol=3 * virt + rng.randint(0, 9), precision=prec,
             roots=rng.randint(1, 2) if kind == "davidson" else 0, dmin=0, dmax=0)
    space = rng.choice(["closed", "empty", "doublet", "triplet"])
    if space == "closed":
        c.update(inactive=rng.randint(4, 20), active=0, act_el=0, mult=1, refs=1)
    elif space == "empty":
        c.update(inactive=rng.randint(4, 8), active=rng.randint(2, 8), act_el=0, mult=1, refs=1)
    elif space == "doublet":
        c.update(inactive=rng.randint(2, 5), active=3, act_el=3, mult=2, refs=rng.randint(1, 3))
    else:
        c.update(inactive=rng.randint(2, 5), active=3, act_el=2, mult=3, refs=rng.randint(1, 2))
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 + seed)


def _operator(case, seed, norb):
    """h and Cholesky vectors of molecular magnitude (numpy, as a program reads them from the integral step)."""
    g = _gen(seed)
    p = torch.repeat_interleave(torch.arange(norb, device="cuda"), torch.arange(1, norb + 1, device="cuda"))
    i = torch.arange(p.numel(), device="cuda")
    q = i - p * (p + 1) // 2
    L = torch.randn(p.numel(), case["nchol"], generator=g, device="cuda", dtype=torch.float64)
    L *= (0.02 * torch.exp(-0.05 * (p - q).double()))[:, None]
    L *= torch.exp(-torch.arange(case["nchol"], device="cuda").double() / 400.0)[None, :]
    h = torch.randn(norb, norb, generator=g, device="cuda", dtype=torch.float64) * 0.02
    h = 0.5 * (h + h.T)
    d = torch.rand(norb, generator=g, device="cuda", dtype=torch.float64) * 3.0 - 2.0
    h[torch.arange(norb), torch.arange(norb)] = torch.sort(d).values
    return h.cpu().numpy(), L.cpu().numpy()


def _references(case):
    """Occupations of the reference configurations over the internal orbitals: the aufbau one, then the top
    doubly occupied active pair moved (or an active electron rotated) up."""
    nact, mult = case["active"], case["mult"]
    docc = (case["act_el"] - (mult - 1)) // 2
    base = [2] * docc + [1] * (mult - 1) + [0] * (nact - docc - mult + 1)
    out = ["2" * case["inactive"] + "".join(map(str, base[k:] + base[:k])) for k in range(case["refs"])]
    return out


def _domains(case):
    """A sorted random subset of the externals for every N-1 and N-2 path of a closed-shell deck."""
    rng = np.random.default_rng(77_000)
    no, n = case["inactive"], case["virt"]

    def doms(k):
        return [np.sort(rng.choice(n, size=int(rng.integers(case["dmin"], case["dmax"] + 1)), replace=False)).tolist()
                for _ in range(k)]

    return doms(no), doms(no * (no + 1) // 2)


def _deck(case):
    nint = case["inactive"] + case["active"]
    nm1, nm2 = _domains(case) if case["dmax"] else (None, None)
    return T.Deck(nint + case["virt"], case["inactive"], case["active"], 2 * case["inactive"] + case["act_el"],
                  case["mult"], _references(case), nm1_domains=nm1, nm2_domains=nm2)


def _chain(case, seed):
    spacing = 1.4 + 1.6 * np.random.default_rng(5_000 + seed).random()
    return serve.request_problem(serve.RequestSpec(0, 0.0, case["atoms"], float(spacing), max(1, case["roots"])),
                                 seed=seed)


def _vector(n, seed):
    c = torch.randn(n, generator=_gen(seed + 7), device="cuda", dtype=torch.float64)
    return c / c.norm()


def _pairs(case):
    return tlocal.pair_domain_problem(case["pairs"], case["n_int"], case["virt"], case["dmin"], case["dmax"], seed=99)


def prepare(case, seed):
    if case["kind"] == "dots":
        small = dict(inactive=3, active=0, act_el=0, mult=1, refs=1, virt=6, nchol=8, dmin=0, dmax=0)
        h, L = _operator(small, 1, 9)
        sb = T.SigmaBuilder(_deck(small), T.Operator(h, L))
        A = torch.randn(case["rows"], case["length"], generator=_gen(seed), device="cuda", dtype=torch.float64)
        return dict(case=case, sb=sb, A=A / A.norm(dim=1, keepdim=True), x=_vector(case["length"], seed),
                    out=torch.zeros(case["rows"], device="cuda", dtype=torch.float64))
    if case["kind"] == "pairs":
        heads, dom, total = _pairs(case)
        _, L = _operator(case, seed, case["n_int"] + case["virt"])
        op = tlocal.LocalAllExternal(case["n_int"], case["virt"], L, heads, dom, total, precision=case["precision"])
        return dict(case=case, op=op, c=_vector(total, seed), s=torch.zeros(total, device="cuda", dtype=torch.float64))
    if case["kind"] == "chain":
        deck, op = _chain(case, seed)
    else:
        deck = _deck(case)
        op = T.Operator(*_operator(case, seed, deck.num_orbitals))
    sb = T.SigmaBuilder(deck, op, precision=case["precision"])
    if case["roots"]:
        return dict(case=case, sb=sb)
    return dict(case=case, sb=sb, c=_vector(sb.n, seed), s=torch.zeros(sb.n, device="cuda", dtype=torch.float64))


def run(state):
    case = state["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "dots":
        A, x = state["A"], state["x"]
        state["sb"].dots(A.data_ptr(), A.stride(0), A.shape[0], x.data_ptr(), x.numel(), state["out"].data_ptr(),
                         stream)
        return state["out"]
    if case.get("roots"):
        # the energies and eigenvectors come back in host memory, as a program that goes on with them has them
        e, v, _ = state["sb"].davidson(case["roots"], tol_residual=1e-6, tol_energy=1e-8, want_vectors=True)
        return {"energies": e, "vectors": v}
    c, s = state["c"], state["s"]
    s.zero_()  # the caller zeroes sigma, as before every htimesc
    if case["kind"] == "pairs":
        state["op"].apply_device(c.data_ptr(), s.data_ptr(), stream)
    else:
        state["sb"].htimesc_device(c.data_ptr(), s.data_ptr(), c.numel(), stream)
    return s


# ---- work -----------------------------------------------------------------------------------------------------

def _sigma_work(no, na, n, heads_s, heads_t, doms=None):
    """Bytes and operations of one sigma build over no occupied (na empty active) orbitals: the CI vectors once
    each way, the integrals once (symmetric halves; on pair domains the (ab|cd) and (ia|bc) blocks of the domains
    only), the contractions on the pairs' own domains."""
    if doms is None:
        ns, nt, m1, m2 = heads_s, heads_t, n, n
        allext = 2.0 * ns * (n * (n + 1) / 2) ** 2 + 2.0 * nt * (n * (n - 1) / 2) ** 2
        dd = 2.0 * (ns + nt) * (no + na) * 2 * float(n) ** 3
        ds = 2 * 2.0 * (ns + nt) * 2 * float(n) ** 3
    else:
        m2 = sum(doms) / len(doms)
        ns, nt, m1 = heads_s, heads_t, m2
        allext = sum((2.0 + (2.0 if k else 0.0)) * (d * d / 2.0) ** 2 for k, d in _head_blocks(doms))
        dd = 2.0 * (ns + nt) * no * 2 * m2 * m2 * m2 * (m2 / n)
        ds = 2 * 2.0 * (ns + nt) * 2 * m2 ** 3
    ci = ns * m2 * (m2 + 1) / 2 + nt * m2 * (m2 - 1) / 2 + no * m1
    integrals = (m2 * (m2 + 1) / 2.0) ** 2 / 2 + no * m2 * m2 * (m2 + 1) / 2.0 + no * no * n * n
    return {"bytes": 8.0 * (3 * ci + integrals), "flops": allext + dd + ds}


def _head_blocks(doms):
    """(the head has a triplet-coupled block, its domain's size) per N-2 head, in the order of the CSF vector."""
    no = (math.isqrt(8 * len(doms) + 1) - 1) // 2
    heads = [(i, j) for i in range(no - 1, -1, -1) for j in range(i, -1, -1)]
    return [(i != j, d) for (i, j), d in zip(heads, doms)]


def work(case):
    if case["kind"] == "dots":
        return {"bytes": 8.0 * (case["rows"] + 1) * case["length"], "flops": 2.0 * case["rows"] * case["length"]}
    if case["kind"] == "pairs":
        heads, dom, total = _pairs(case)
        flops = sum(4.0 * case["nchol"] * hd[2] * float(hd[6]) ** 3 for hd in heads)
        n = case["virt"]
        return {"bytes": 8.0 * (3 * total + n * (n + 1) // 2 * case["nchol"]), "flops": flops}
    if case["kind"] == "chain":
        no, na, n = case["atoms"] // 2, 1, 5 * case["atoms"] - case["atoms"] // 2 - 1
    else:
        no, na, n = case["inactive"] + (case["act_el"] + 1) // 2, case["active"], case["virt"]
        na -= (case["act_el"] + 1) // 2
    doms = [len(d) for d in _domains(case)[1]] if case.get("dmax") else None
    w = _sigma_work(no, na, n, no * (no + 1) // 2, no * (no - 1) // 2, doms)
    if case["roots"]:  # a solve builds sigma at least a few times per root; the integrals are read every time
        w = {k: 8 * case["roots"] * v for k, v in w.items()}
    return w


# ---- exact results in 64 bits ---------------------------------------------------------------------------------

def _closed_shell_sigma(h, L, no, n, c, nm1, nm2):
    """H c of a closed-shell singles-and-doubles CI in spin-free amplitudes (T[i,j,a,b]: i alpha -> a alpha with
    j beta -> b beta), on the CSF order valence, N-1 heads (the highest hole first), N-2 heads (holes i >= j, the
    highest first): aa block, then the singlet-coupled and the triplet-coupled pairs a > b; nm1, nm2: the heads'
    sorted domains in that order."""
    dev, f8 = "cuda", torch.float64
    norb = no + n
    Lf = torch.empty(norb, norb, L.shape[1], dtype=f8, device=dev)
    p, q = np.tril_indices(norb)
    Lf[p, q] = Lf[q, p] = torch.as_tensor(L, device=dev)
    h = torch.as_tensor(h, device=dev)
    o, v = slice(0, no), slice(no, norb)
    Loo, Lov, Lvv = Lf[o, o].contiguous(), Lf[o, v].contiguous(), Lf[v, v].permute(2, 0, 1).contiguous()
    f = h + 2 * torch.einsum("pqJ,J->pq", Lf, torch.einsum("kkJ->J", Loo)) - torch.einsum(
        "pkJ,qkJ->pq", Lf[:, o], Lf[:, o])
    e0 = float(torch.diagonal(h + f)[:no].sum())
    del Lf
    # amplitudes from the CSF coefficients
    T2 = torch.zeros(no, no, n, n, dtype=f8, device=dev)
    t = torch.zeros(no, n, dtype=f8, device=dev)
    c0, at = c[0], 1
    where = []
    for lex in range(no):
        i, d = no - 1 - lex, torch.as_tensor(nm1[lex], device=dev)
        where.append((at, i, d))
        t[i, d] = c[at:at + len(d)] / math.sqrt(2.0)
        at += len(d)
    pairs = []
    for i in range(no - 1, -1, -1):
        for j in range(i, -1, -1):
            d = torch.as_tensor(nm2[len(pairs)], device=dev)
            m = len(d)
            x, y = torch.tril_indices(m, m, -1, device=dev)
            nab = x.numel()
            pairs.append((i, j, d, x, y, at))
            D = torch.zeros(m, m, dtype=f8, device=dev)
            D[torch.arange(m), torch.arange(m)] = math.sqrt(2.0) * c[at:at + m]
            D[x, y] = D[y, x] = c[at + m:at + m + nab]
            if i == j:
                T2[i, i][d[:, None], d] = D / math.sqrt(2.0)
            else:
                E = torch.zeros(m, m, dtype=f8, device=dev)
                E[x, y] = c[at + m + nab:at + m + 2 * nab]
                E = E - E.T
                B = -D / 2 - E / (2 * math.sqrt(3.0))
                T2[i, j][d[:, None], d] = B
                T2[j, i][d[:, None], d] = B.T
            at += m + (1 if i == j else 2) * nab
    assert at == c.numel()
    J = torch.einsum("ijP,Pab->ijab", Loo, Lvv)          # (ij|ab)
    K = torch.einsum("iaP,jbP->iajb", Lov, Lov)          # (ia|jb)
    U = 2 * T2 - T2.transpose(2, 3)
    s0 = e0 * c0 + 2 * (f[o, v] * t).sum() + torch.einsum("iajb,ijab->", K, U)
    s1 = e0 * t + f[o, v] * c0 + t @ f[v, v] - f[o, o] @ t
    s1 += 2 * torch.einsum("iajb,jb->ia", K, t) - torch.einsum("ijab,jb->ia", J, t)
    s1 += torch.einsum("jb,ijab->ia", f[o, v], U)
    s1 -= torch.einsum("jiP,kbP,jkab->ia", Loo, Lov, U)
    # one half of the doubles; the other is its transpose under (ia) <-> (jb)
    R = torch.einsum("ia,jb->ijab", f[o, v], t)
    R += torch.einsum("ijac,bc->ijab", T2, f[v, v]) - torch.einsum("kj,ikab->ijab", f[o, o], T2)
    R += torch.einsum("ikac,kcjb->ijab", U, K) - torch.einsum("kjbc,ikac->ijab", J, T2)
    R -= torch.einsum("kjac,ikcb->ijab", J, T2)
    R -= torch.einsum("kiP,jbP,ka->ijab", Loo, Lov, t)
    Up = U.permute(0, 2, 1, 3).reshape(no * n, no * n)
    tmp = torch.zeros(no, n, L.shape[1], dtype=f8, device=dev)   # sum_jc (jc|P) U_ij^bc
    tmp = (Up @ Lov.reshape(no * n, -1)).reshape(no, n, -1)
    s1 += torch.einsum("Pab,ibP->ia", Lvv, tmp)
    Lt = torch.einsum("Pac,ic->iaP", Lvv, t)
    R += torch.einsum("iaP,jbP->ijab", Lt, Lov)                   # (ac|bj) t_i^c
    R = R + R.permute(1, 0, 3, 2)
    R += e0 * T2 + c0 * K.permute(0, 2, 1, 3)
    oooo = torch.einsum("kiP,ljP->kilj", Loo, Loo)
    R += torch.einsum("kilj,klab->ijab", oooo, T2)
    for i, j, d, x, y, _ in pairs:                                # (ac|bd) T_ij^cd on the pair's domain
        m = len(d)
        B = T2[i, j][d[:, None], d]
        S = torch.zeros(m, m, dtype=f8, device=dev)
        for k in range(0, L.shape[1], 256):
            Lk = Lvv[k:k + 256][:, d[:, None], d]
            S += torch.einsum("Pae,Peb->ab", Lk @ B, Lk) if m < 8 else \
                ((Lk @ B).permute(1, 0, 2).reshape(m, -1) @ Lk.reshape(-1, m))
        R[i, j][d[:, None], d] += S
    out = torch.zeros_like(c)
    out[0] = s0
    for a0, i, d in where:
        out[a0:a0 + len(d)] = math.sqrt(2.0) * s1[i, d]
    for i, j, d, x, y, a0 in pairs:
        B = R[i, j][d[:, None], d]
        m, nab = len(d), x.numel()
        w = 1.0 if i == j else -math.sqrt(2.0)
        out[a0:a0 + m] = w * torch.diagonal(B)
        S = (B + B.T) * (math.sqrt(0.5) if i == j else -1.0)
        out[a0 + m:a0 + m + nab] = S[x, y]
        if i != j:
            A = -math.sqrt(3.0) * (B - B.T)
            out[a0 + m + nab:a0 + m + 2 * nab] = A[x, y]
    return out


def exact(case, seed):
    if case["kind"] == "dots":
        A = torch.randn(case["rows"], case["length"], generator=_gen(seed), device="cuda", dtype=torch.float64)
        return (A / A.norm(dim=1, keepdim=True)) @ _vector(case["length"], seed)
    if case["kind"] == "pairs":
        heads, dom, total = _pairs(case)
        _, L = _operator(case, seed, case["n_int"] + case["virt"])
        c = _vector(total, seed)
        n, no = case["virt"], case["n_int"]
        p, q = np.tril_indices(n)
        rows = (p + no) * (p + no + 1) // 2 + q + no
        Lvv = torch.zeros(case["nchol"], n, n, dtype=torch.float64, device="cuda")
        Lvv[:, p, q] = Lvv[:, q, p] = torch.as_tensor(L[rows], device="cuda").T
        out = torch.zeros_like(c)
        for ab, aa, nsf, naa, nsing, o, m in heads.tolist():
            d = torch.as_tensor(dom[o:o + m], device="cuda")
            x, y = torch.tril_indices(m, m, -1, device="cuda")
            for k in range(nsf):
                sgn = 1.0 if k < nsing else -1.0
                at = ab + k * x.numel()
                D = torch.zeros(m, m, dtype=torch.float64, device="cuda")
                D[x, y] = sgn * c[at:at + x.numel()]
                D[y, x] = c[at:at + x.numel()]
                if k < naa:
                    D[torch.arange(m), torch.arange(m)] = math.sqrt(2.0) * c[aa:aa + m]
                S = torch.zeros_like(D)
                for j in range(0, case["nchol"], 128):
                    Lk = Lvv[j:j + 128][:, d[:, None], d]
                    S += (Lk @ D).permute(1, 0, 2).reshape(m, -1) @ Lk.reshape(-1, m)
                out[at:at + x.numel()] = S[y, x]
                if k < naa:
                    out[aa:aa + m] = torch.diagonal(S) / math.sqrt(2.0)
        return out
    if case["kind"] == "sigma" and not case["roots"] and not case["active"]:
        no, n = case["inactive"], case["virt"]
        h, L = _operator(case, seed, no + n)
        if case["dmax"]:
            nm1, nm2 = _domains(case)
        else:
            nm1, nm2 = [list(range(n))] * no, [list(range(n))] * (no * (no + 1) // 2)
        total = 1 + sum(len(d) for d in nm1)
        for off, m in _head_blocks([len(d) for d in nm2]):
            total += m + (2 if off else 1) * (m * (m - 1) // 2)
        return _closed_shell_sigma(h, L, no, n, _vector(total, seed), nm1, nm2)
    return None  # several references or open shells: the order and phases of the CSFs have no short statement
