"""The work a quantum-chemistry program has this library do, as measurable cases.

One pass is one Fock build (closed shell, mixed precision, open shell or a
batch of molecules) or one Schwarz table, through the library's Python front
end.  A program sets a handle up once per geometry and then builds F from a
new density in every SCF iteration, so the handle belongs to ``prepare`` and
the build to ``run``.

Molecules are the synthetic ones of ``gms_liberi_b200.molecules``.  A case
names its kind and size, ``geom`` picks composition and positions; the seed
moves every atom by a few hundredths of a bohr (as the steps of a geometry
optimisation do) and makes the density.
"""
import math

import numpy as np
import torch

from gms_liberi_b200 import flops
from gms_liberi_b200 import liberi
from gms_liberi_b200 import molecules as M

CUT = 5.00000000000000018e-11  # the library's default Schwarz cut and integral cut
_NCART = (1, 3, 6, 10)


# ---- cases ----------------------------------------------------------------------
def listed():
    return [
        # The smallest call there is: a triatomic in a minimal basis, host
        # arrays in and out, as a program linked against the handle API has it.
        # Latency and launches are all it has.
        {"name": "water_min_host", "op": "fock", "mol": "water", "natoms": 3, "geom": 0, "api": "host"},
        # A small organic molecule with d shells, the same drop-in call.
        {"name": "ethane_host", "op": "fock", "mol": "ethane", "natoms": 8, "geom": 0, "api": "host"},
        # A 10-atom molecule in the mixed tier on device buffers: what a
        # serving loop's smallest session runs.
        {"name": "mol10_mixed", "op": "fock", "mol": "random", "natoms": 10, "geom": 3, "api": "device",
         "fp32_cut": 1e-5},
        # An open-shell build (two F from two densities) of an odd-sized molecule.
        {"name": "mol17_uhf_host", "op": "uhf", "mol": "random", "natoms": 17, "geom": 1, "api": "host"},
        # An ordinary molecule, FP64, device buffers.
        {"name": "mol40", "op": "fock", "mol": "random", "natoms": 40, "geom": 0, "api": "device"},
        # f shells, small: three atoms that fill all 34 f classes.
        {"name": "f_triatomic_host", "op": "fock", "mol": "f_triatomic", "natoms": 3, "geom": 0, "api": "host"},
        # f polarisation shells on every heavy atom of a 30-atom cluster.
        {"name": "f_cluster30", "op": "fock", "mol": "f_cluster", "natoms": 30, "geom": 0, "api": "device"},
        # Many small molecules in one captured graph per SCF iteration, FP64.
        {"name": "batch40", "op": "batch", "mol": "random", "natoms": 40, "count": 40, "geom": 0},
        # A large serving session: 100 atoms, mixed at the serving cut.
        {"name": "mol100_mixed", "op": "fock", "mol": "random", "natoms": 100, "geom": 0, "api": "device",
         "fp32_cut": 1e-7},
        # The headline molecule in the mixed tier, and in FP64 (the largest).
        {"name": "c60_mixed", "op": "fock", "mol": "c60", "natoms": 60, "geom": 0, "api": "device",
         "fp32_cut": 1e-5},
        {"name": "c60", "op": "fock", "mol": "c60", "natoms": 60, "geom": 0, "api": "device"},
        # The Schwarz table a program without its own asks for once per geometry.
        {"name": "schwarz40", "op": "schwarz", "mol": "random", "natoms": 40, "geom": 0},
    ]


def draw(rng):
    """Builds of 3 to 70 atoms in every tier, f clusters of 3 to 24 atoms,
    batches of 3 to 36 molecules and Schwarz tables."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    geom = rng.randrange(1, 1000)
    op = rng.choice(["fock", "fock", "mixed", "mixed", "uhf", "f", "batch", "batch_mixed", "schwarz"])
    api = rng.choice(["host", "device"])
    cut = rng.choice([1e-4, 1e-5, 1e-6, 1e-7, 1e-8])
    if op == "fock":
        return {"op": "fock", "mol": "random", "natoms": size(3, 70), "geom": geom, "api": api}
    if op == "mixed":
        return {"op": "fock", "mol": "random", "natoms": size(3, 80), "geom": geom, "api": api, "fp32_cut": cut}
    if op == "uhf":
        return {"op": "uhf", "mol": "random", "natoms": size(3, 50), "geom": geom, "api": "host"}
    if op == "f":
        return {"op": "fock", "mol": "f_cluster", "natoms": size(3, 24), "geom": geom, "api": api}
    if op == "batch":
        return {"op": "batch", "mol": "random", "natoms": size(6, 40), "count": size(3, 36), "geom": geom}
    if op == "batch_mixed":
        return {"op": "batch", "mol": "random", "natoms": size(6, 40), "count": size(3, 36), "geom": geom,
                "fp32_cut": cut}
    return {"op": "schwarz", "mol": rng.choice(["random", "f_cluster"]), "natoms": size(3, 40), "geom": geom}


# ---- inputs ---------------------------------------------------------------------
def _basis(mol, natoms, geom, seed=None):
    if mol == "water":
        b = M.h2o_like()
    elif mol == "ethane":
        b = M.ethane()
    elif mol == "c60":
        b = M.c60()
    elif mol == "f_triatomic":
        b = M.f_triatomic()
    elif mol == "f_cluster":
        b = M.f_cluster(natoms, geom)
    else:
        b = M.random_molecule(natoms, geom)
    if seed is not None:
        rng = np.random.default_rng([seed, natoms, geom])
        b["coords"] = b["coords"] + 0.02 * rng.standard_normal(b["coords"].size)
    return b


def _members(case, seed=None):
    """The molecules of a batch: 3 to ``natoms`` atoms each, evenly spread."""
    n, top = case["count"], case["natoms"]
    return [_basis("random", 3 + round((top - 3) * i / max(1, n - 1)), case["geom"] + i, seed) for i in range(n)]


def _density(b, seed, spin=0):
    nocc = min(b["num_bas"], max(1, M.nocc_of(b) + (spin == 1)))
    d = M.density(b["num_bas"], nocc, [seed, b["num_bas"], spin])
    return d if spin == 0 else 0.5 * d


def _handle(case, b):
    h = liberi.liberi_create()
    if "fp32_cut" in case:
        h.set_option("precision", 1)
        h.set_option("fp32_cut", case["fp32_cut"])
    liberi.setup_from_basis(h, b, liberi.schwarz(b))
    return h


def prepare(case, seed):
    if case["op"] == "batch":
        bs = _members(case, seed)
        hs = [_handle(case, b) for b in bs]
        D = [torch.from_numpy(_density(b, seed)).cuda() for b in bs]
        F = [torch.empty_like(d) for d in D]
        batch = liberi.Batch(hs)
        batch.bind([d.data_ptr() for d in D], [f.data_ptr() for f in F])
        batch.capture()
        return {"op": "batch", "batch": batch, "D": D, "F": F, "stream": torch.cuda.Stream()}
    b = _basis(case["mol"], case["natoms"], case["geom"], seed)
    if case["op"] == "schwarz":
        return {"op": "schwarz", "basis": b}
    h = _handle(case, b)
    dens = [_density(b, seed, s) for s in ((1, 2) if case["op"] == "uhf" else (0,))]
    st = {"op": case["op"], "api": case["api"], "handle": h}
    if case["api"] == "host":
        st["D"] = dens
    else:
        st["D"] = [torch.from_numpy(d).cuda() for d in dens]
        st["F"] = [torch.empty_like(d) for d in st["D"]]
        st["stream"] = torch.cuda.Stream()
    return st


def run(state):
    op = state["op"]
    if op == "schwarz":
        return liberi.schwarz(state["basis"])
    if op != "batch" and state["api"] == "host":
        if op == "uhf":
            return list(liberi.fock_uhf(state["handle"], *state["D"]))
        return liberi.fock(state["handle"], state["D"][0])
    # device buffers: the build is enqueued on the program's own stream
    cur, st = torch.cuda.current_stream(), state["stream"]
    st.wait_stream(cur)
    D, F = state["D"], state["F"]
    if op == "batch":
        state["batch"].launch(st.cuda_stream)
    else:
        liberi.fock_build_device(state["handle"], D[0].data_ptr(), F[0].data_ptr(), st.cuda_stream)
    cur.wait_stream(st)
    return F


# ---- what a pass cannot do without ----------------------------------------------
def _shells(b):
    xyz = np.asarray(b["coords"]).reshape(-1, 3)
    out, bf = [], 0
    for s in range(b["nsh"]):
        l, lo, k = b["ang_mom"][s] - 1, b["sh_loc"][s] - 1, b["contr_num"][s]
        c = (b["coef_s"], b["coef_p"], b["coef_d"], b["coef_f"])[l][lo:lo + k]
        out.append((l, bf, xyz[b["atom_num"][s] - 1], np.asarray(b["exponents"][lo:lo + k]), np.asarray(c)))
        bf += _NCART[l]
    return out


def _pair_sizes(b):
    """Per (la, lb) with la >= lb: size estimate of every shell pair's
    sqrt((ab|ab)) from its primitives' s-type charge distributions, and its
    number of primitive pairs."""
    sh = _shells(b)
    out = {}
    for i, (li, _, ri, ei, ci) in enumerate(sh):
        for (lj, _, rj, ej, cj) in sh[:i + 1]:
            p = ei[:, None] + ej[None, :]
            r2 = float(((ri - rj) ** 2).sum())
            mu = ei[:, None] * ej[None, :] / p
            width = 1.0 / np.sqrt(2.0 * p)
            reach = (np.sqrt(r2) * ej[None, :] / p + width) ** li * (np.sqrt(r2) * ei[:, None] / p + width) ** lj
            q = np.abs(ci[:, None] * cj[None, :]) * np.exp(-mu * r2) * (math.pi / p) ** 1.5 * (2 * p / math.pi) ** 0.25
            out.setdefault((max(li, lj), min(li, lj)), []).append(
                (float((q * reach).sum()), int((mu * r2 <= 50.0).sum())))
    return {k: np.array(sorted(v, reverse=True)) for k, v in out.items()}


def _build_flops(b):
    """Operations of one build: primitive quartets of the shell quartets whose
    estimated Schwarz product passes the cut, at the library's counted cost."""
    cls = _pair_sizes(b)
    keys = sorted(cls)
    total = 0.0
    for i, bra in enumerate(keys):
        for ket in keys[:i + 1]:
            A, B = cls[bra], cls[ket]
            c_prim, c_shell = flops.engine_costs(*bra, *ket)
            n = np.searchsorted(-B[:, 0], -(CUT / np.maximum(A[:, 0], 1e-300)), side="left")
            cum = np.concatenate([[0.0], np.cumsum(B[:, 1])])
            nprim, nshell = float((A[:, 1] * cum[n]).sum()), float(n.sum())
            total += (c_prim * nprim + c_shell * nshell) * (0.5 if bra == ket else 1.0)
    return total


def work(case):
    bs = _members(case) if case["op"] == "batch" else [_basis(case["mol"], case["natoms"], case["geom"])]
    byt = flo = 0.0
    for b in bs:
        prims = 8.0 * 2 * float(np.sum(b["contr_num"])) + 8.0 * 3 * b["natoms"]
        tri = b["num_bas"] * (b["num_bas"] + 1) / 2
        shtri = b["nsh"] * (b["nsh"] + 1) / 2
        if case["op"] == "schwarz":
            byt += prims + 8.0 * shtri
            for (la, lb), v in _pair_sizes(b).items():
                flo += float((v[:, 1] ** 2).sum()) * flops.engine_costs(la, lb, la, lb)[0]
        else:
            nf = 2 if case["op"] == "uhf" else 1  # densities in, Fock matrices out
            byt += prims + 8.0 * shtri + nf * 2 * 8.0 * tri
            # the integrals of an open-shell build serve both spins; its second digestion is left out
            flo += _build_flops(b)
    return {"bytes": byt, "flops": flo}


def tolerance(case):
    # FP64: against ``exact`` the builds show 1e-15 to 2e-12 in the 2-norm (the
    # most where integrals lie at the integral cut), f shells 9e-14.  Mixed:
    # quartets below fp32_cut / max|D| are single precision, so the error goes
    # with the cut; against FP64 builds of 10 to 100 atoms and C60 it is up to
    # 1.8e-10, 4.5e-11, 8.6e-12, 1.4e-12 and 2.4e-13 at cuts 1e-4 to 1e-8.
    if case["op"] == "schwarz":
        return {"rel": 1e-12}
    return {"rel": 5e-12 + 3e-5 * case.get("fp32_cut", 0.0)}


# ---- the same in 64 bits, without the library -----------------------------------
# McMurchie-Davidson: every primitive pair's Cartesian products expanded in
# Hermite Gaussians, Coulomb integrals between those from the Boys function.
_CART = {0: [(0, 0, 0)],
         1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
         2: [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)],
         3: [(3, 0, 0), (0, 3, 0), (0, 0, 3), (2, 1, 0), (2, 0, 1), (1, 2, 0), (0, 2, 1), (1, 0, 2), (0, 1, 2),
             (1, 1, 1)]}


def _dfact(n):
    return 1.0 if n <= 0 else n * _dfact(n - 2)


def _norm(l, e):
    """Component norm relative to the axial one: sqrt((2l-1)!! / prod (2e-1)!!)."""
    return math.sqrt(_dfact(2 * l - 1) / (_dfact(2 * e[0] - 1) * _dfact(2 * e[1] - 1) * _dfact(2 * e[2] - 1)))


def _herm(l):
    return [(t, u, l2 - t - u) for l2 in range(l + 1) for t in range(l2 + 1) for u in range(l2 - t + 1)]


def _boys(n, T):
    """F_0..F_n(T): positive series and downward recursion below T = 35, erf
    and upward recursion above."""
    out = torch.empty((n + 1,) + T.shape, dtype=T.dtype, device=T.device)
    Ts = T.clamp(max=35.0)
    ex = torch.exp(-Ts)
    term = torch.full_like(T, 1.0 / (2 * n + 1))
    s = term.clone()
    for k in range(1, 160):
        term = term * (2.0 * Ts / (2 * n + 2 * k + 1))
        s = s + term
    low = ex * s
    out[n] = low
    for m in range(n - 1, -1, -1):
        low = (2.0 * Ts * low + ex) / (2 * m + 1)
        out[m] = low
    big = T > 35.0
    Tb = T.clamp(min=35.0)
    up = 0.5 * torch.sqrt(math.pi / Tb) * torch.erf(torch.sqrt(Tb))
    exb = torch.exp(-Tb)
    for m in range(n + 1):
        out[m] = torch.where(big, up, out[m])
        up = ((2 * m + 1) * up - exb) / (2.0 * Tb)
    return out


def _pair_class(sh, la, lb, dev):
    """Primitive pairs of the shell pairs (la, lb): exponent, centre, Hermite
    expansion [nprim, ncomp, nherm] (coefficients and norms in), owner pair,
    and per shell pair its first functions."""
    P, C, RA, RB, EA, EB, own, bf = [], [], [], [], [], [], [], []
    for i, (li, bi, ri, ei, ci) in enumerate(sh):
        for j, (lj, bj, rj, ej, cj) in enumerate(sh):
            if li != la or lj != lb or (la == lb and j > i):
                continue
            for a, ca in zip(ei, ci):
                for b, cb in zip(ej, cj):
                    own.append(len(bf))
                    EA.append(a)
                    EB.append(b)
                    C.append(ca * cb)
                    RA.append(ri)
                    RB.append(rj)
            bf.append((bi, bj))
    if not bf:
        return None
    t = lambda x: torch.tensor(np.array(x), dtype=torch.float64, device=dev)  # noqa: E731
    a, b, c, ra, rb = t(EA), t(EB), t(C), t(RA), t(RB)
    p = a + b
    ctr = (a[:, None] * ra + b[:, None] * rb) / p[:, None]
    c = c * torch.exp(-a * b / p * ((ra - rb) ** 2).sum(1))
    e1 = []
    for x in range(3):  # E[i][j][t] of one axis
        pa, pb = ctr[:, x] - ra[:, x], ctr[:, x] - rb[:, x]
        E = {(0, 0): [torch.ones_like(p)]}
        step = lambda o, d: [(o[k - 1] / (2 * p) if k else 0.0) + (d * o[k] if k < len(o) else 0.0) +  # noqa: E731
                             ((k + 1) * o[k + 1] if k + 1 < len(o) else 0.0) for k in range(len(o) + 1)]
        for i in range(la + 1):
            if i:
                E[i, 0] = step(E[i - 1, 0], pa)
            for j in range(1, lb + 1):
                E[i, j] = step(E[i, j - 1], pb)
        e1.append(E)
    hs = _herm(la + lb)
    out = torch.zeros(len(own), _NCART[la] * _NCART[lb], len(hs), dtype=torch.float64, device=dev)
    for ia, ca in enumerate(_CART[la]):
        for ib, cb in enumerate(_CART[lb]):
            nrm = _norm(la, ca) * _norm(lb, cb)
            for k, h in enumerate(hs):
                ex = [e1[x][ca[x], cb[x]] for x in range(3)]
                if all(h[x] < len(ex[x]) for x in range(3)):
                    out[:, ia * _NCART[lb] + ib, k] = nrm * c * ex[0][h[0]] * ex[1][h[1]] * ex[2][h[2]]
    return {"p": p, "R": ctr, "E": out, "own": torch.tensor(own, device=dev), "n": len(bf), "bf": bf, "L": la + lb}


def _hermite_coulomb(L, alpha, d):
    """R_{tuv} for t+u+v <= L: alpha and d[..., 3] of every primitive quartet."""
    F = _boys(L, alpha * (d * d).sum(-1))
    R = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * F[n]}
        for (t, u, v) in _herm(L - n):
            if t:
                new[t, u, v] = d[..., 0] * R[t - 1, u, v] + ((t - 1) * R[t - 2, u, v] if t > 1 else 0.0)
            elif u:
                new[t, u, v] = d[..., 1] * R[t, u - 1, v] + ((u - 1) * R[t, u - 2, v] if u > 1 else 0.0)
            elif v:
                new[t, u, v] = d[..., 2] * R[t, u, v - 1] + ((v - 1) * R[t, u, v - 2] if v > 1 else 0.0)
        R = new
    return R


def _eri(bra, ket):
    """[bra pairs, ket pairs, bra comps, ket comps] contracted integrals."""
    hb, hk = _herm(bra["L"]), _herm(ket["L"])
    dev = bra["p"].device
    out = torch.zeros(bra["n"], ket["n"], bra["E"].shape[1], ket["E"].shape[1], dtype=torch.float64, device=dev)
    nq = ket["p"].numel()
    per = nq * (len(hb) * len(hk) + 12 * (bra["L"] + ket["L"] + 1) + len(_herm(bra["L"] + ket["L"])))
    chunk = max(1, int(6e7 // per))
    sign = [(-1.0) ** sum(k) for k in hk]
    for s in range(0, bra["p"].numel(), chunk):
        p, q = bra["p"][s:s + chunk, None], ket["p"][None, :]
        d = bra["R"][s:s + chunk, None, :] - ket["R"][None, :, :]
        R = _hermite_coulomb(bra["L"] + ket["L"], p * q / (p + q), d)
        pref = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        H = torch.stack([torch.stack([sg * pref * R[a[0] + b[0], a[1] + b[1], a[2] + b[2]]
                                      for b, sg in zip(hk, sign)], -1) for a in hb], -2)  # [p, q, h, k]
        Y = torch.einsum("pqhk,qbk->qphb", H, ket["E"])
        Yc = torch.zeros((ket["n"],) + Y.shape[1:], dtype=torch.float64, device=dev).index_add_(0, ket["own"], Y)
        Z = torch.einsum("pah,Qphb->pQab", bra["E"][s:s + chunk], Yc)
        out.index_add_(0, bra["own"][s:s + chunk], Z)
    return out


def _full_eri(b, dev):
    """(ij|kl) over all functions as an [n^2, n^2] matrix, integrals below the cut dropped."""
    n, sh = b["num_bas"], _shells(b)
    G = torch.zeros(n * n, n * n, dtype=torch.float64, device=dev)
    cls = [c for c in (_pair_class(sh, la, lb, dev) for la in range(4) for lb in range(la + 1)) if c]

    def index(c, flip):
        out = []
        for (bi, bj) in c["bf"]:
            na = _NCART[[s[0] for s in sh if s[1] == bi][0]]
            nb = _NCART[[s[0] for s in sh if s[1] == bj][0]]
            i, j = np.meshgrid(np.arange(bi, bi + na), np.arange(bj, bj + nb), indexing="ij")
            out.append(((j * n + i) if flip else (i * n + j)).reshape(-1))
        return torch.tensor(np.array(out), device=dev)

    for x, bra in enumerate(cls):
        for ket in cls[:x + 1]:
            v = _eri(bra, ket)
            v = torch.where(v.abs() < CUT, torch.zeros_like(v), v).permute(0, 2, 1, 3)
            m = v.reshape(v.shape[0] * v.shape[1], -1)
            for f in (False, True):
                for g in (False, True):
                    r, c = index(bra, f).reshape(-1), index(ket, g).reshape(-1)
                    G[r[:, None], c[None, :]] = m
                    G[c[:, None], r[None, :]] = m.T
    return G


def _fock_exact(G, n, Dj, Dk):
    """Packed J(Dj) - K(Dk) in the library's units: twice J - K/2, the diagonal once."""
    J = (G @ Dj.reshape(-1)).reshape(n, n)
    K = torch.einsum("ijkl,jl->ik", G.view(n, n, n, n), Dk)
    F = 2.0 * J - K
    F.diagonal().mul_(0.5)
    return M.pack(F.cpu().numpy())


def _schwarz_exact(b, dev):
    """sqrt(max over components |(ab|ab)|) of every shell pair, packed."""
    sh, nsh = _shells(b), b["nsh"]
    of_bf = {s[1]: i for i, s in enumerate(sh)}
    out = np.zeros(nsh * (nsh + 1) // 2)
    for la in range(4):
        for lb in range(la + 1):
            c = _pair_class(sh, la, lb, dev)
            if not c:
                continue
            count = torch.bincount(c["own"], minlength=c["n"])
            first = torch.cumsum(count, 0) - count
            herm = _herm(c["L"])
            for K in count.unique().tolist():
                pairs = (count == K).nonzero()[:, 0]
                step = max(1, int(3e7 // (K * K * (len(herm) ** 2 + len(_herm(2 * c["L"])) + 40))))
                for s in range(0, pairs.numel(), step):
                    some = pairs[s:s + step]
                    rows = first[some][:, None] + torch.arange(K, device=dev)
                    p, R3, E = c["p"][rows], c["R"][rows], c["E"][rows]
                    pp, qq = p[:, :, None], p[:, None, :]
                    R = _hermite_coulomb(2 * c["L"], pp * qq / (pp + qq), R3[:, :, None] - R3[:, None, :])
                    pref = 2.0 * math.pi ** 2.5 / (pp * qq * torch.sqrt(pp + qq))
                    H = torch.stack([torch.stack([(-1.0) ** sum(k) * pref * R[a[0] + k[0], a[1] + k[1], a[2] + k[2]]
                                                  for k in herm], -1) for a in herm], -2)
                    v = torch.einsum("npah,npqhk,nqak->na", E, H, E).abs().amax(1).sqrt().cpu().numpy()
                    for x, pair in zip(v, some.tolist()):
                        i, j = (of_bf[f] for f in c["bf"][pair])
                        i, j = max(i, j), min(i, j)
                        out[i * (i + 1) // 2 + j] = x
    return out


def exact(case, seed):
    if case["op"] == "batch":
        return None
    b = _basis(case["mol"], case["natoms"], case["geom"], seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["op"] == "schwarz":
        return _schwarz_exact(b, dev) if b["nsh"] <= 200 else None
    n = b["num_bas"]
    if n > 80:
        return None
    G = _full_eri(b, dev)
    dens = [_density(b, seed, s) for s in ((1, 2) if case["op"] == "uhf" else (0,))]
    D = [torch.from_numpy(M.unpack(d, n)).to(dev) for d in dens]
    if case["op"] == "uhf":
        return [_fock_exact(G, n, D[0] + D[1], 2.0 * d) for d in D]
    F = _fock_exact(G, n, D[0], D[0])
    return F if case["api"] == "host" else [F]
