"""The workloads whose speed is followed from one version of the library to the next.

``listed()`` names them, ``draw(rng)`` gives further ones of the same ranges,
``prepare(case, seed)`` makes a case's inputs (and the plan that a program keeps),
``run(state)`` is one pass through the public entry points, ``work(case)`` the bytes and
operations that a pass cannot do without, and ``exact(case, seed)`` its result as plain
torch gives it in 64 bits.

The kinds of cases are the calls a density-functional program makes:

``gemm``    C += op(A) op(B), f64 or f32 data, FP64 or split precision, any transposes
            and row strides, on device tensors
``masked``  the masked GEMM, B's (row, column block) tiles present or absent
``rho``     the masked AO-DM-AO contraction (the electron density), on device tensors
``host``    the same contraction on numpy arrays, as the drop-in replacement is called
``fock``    the transpose contraction (the potential's matrix elements)
``plan``    many uneven grid batches of one molecule, one plan kept and run per step

Every output is accumulated into by the library, so a pass clears it first, as a
program that wants the plain result does.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

cm = importlib.import_module("cfgable-matmul_b200")

BOHR = 0.529177210903


def listed():
    return [
        # the smallest products: overlap blocks, one shell pair; latency and launches
        dict(name="gemm_small", kind="gemm", dtype="f64", prec="fp64", m=131, n=257, k=300,
             transa=False, transb=False, pad=0),
        # an ordinary product of odd sizes, both operands transposed, padded rows
        dict(name="gemm_odd_tt", kind="gemm", dtype="f64", prec="fp64", m=1021, n=1537, k=1999,
             transa=True, transb=True, pad=3),
        # the large product that the library's benchmark is quoted on, FP64 ...
        dict(name="gemm_full", kind="gemm", dtype="f64", prec="fp64", m=3527, n=9583, k=6581,
             transa=False, transb=False, pad=0),
        # ... and in split precision
        dict(name="gemm_full_split", kind="gemm", dtype="f64", prec="split", m=3527, n=9583,
             k=6581, transa=False, transb=False, pad=0),
        # single-precision data of ordinary size, split precision, A transposed
        dict(name="gemm_f32_split", kind="gemm", dtype="f32", prec="split", m=1111, n=2228,
             k=3001, transa=True, transb=False, pad=0),
        # X = D phi with the reference's own test shape and tile density
        dict(name="masked_gemm", kind="masked", prec="fp64", m=2228, n=16384, k=2228,
             transa=False, blk=48, density=0.3),
        # a small molecule's density on one batch of points, a few tens of microseconds
        dict(name="rho_small", kind="rho", prec="fp64", nao=512, ngrid=4096, nset=1, blk=64,
             density=0.3, mask="bernoulli"),
        # the density of a drug-size molecule, three density matrices, FP64 ...
        dict(name="rho_taxol", kind="rho", prec="fp64", nao=2228, ngrid=16384, nset=3, blk=64,
             density=0.3, mask="centres"),
        # ... and in split precision
        dict(name="rho_taxol_split", kind="rho", prec="split", nao=2228, ngrid=16384, nset=3,
             blk=64, density=0.3, mask="centres"),
        # the step after it: the potential's matrix elements on the same grid
        dict(name="fock_taxol", kind="fock", nao=2228, ngrid=16384, nset=3, blk=64, density=0.3,
             mask="centres"),
        # an SCF step over a whole uneven grid: the plan is kept, D changes
        dict(name="plan_uneven", kind="plan", prec="split", nao=2228, nbatch=256, gmin=128,
             gmax=4096, dmin=0.05, dmax=0.6, nset=3, blk=64),
        # the drop-in call on host memory, blocks of 48 points, a ragged last one
        dict(name="rho_host", kind="host", nao=601, ngrid=8191, nset=1, blk=48, density=0.3,
             mask="centres"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "masked", "rho", "rho", "fock", "plan", "host"])
    if kind == "gemm":
        m, n, k = _log_int(rng, 100, 3527), _log_int(rng, 100, 9583), _log_int(rng, 100, 6581)
        return dict(kind=kind, dtype=rng.choice(["f64", "f64", "f32"]),
                    prec=rng.choice(["fp64", "split"]), m=m, n=n, k=k,
                    transa=rng.random() < 0.5, transb=rng.random() < 0.5,
                    pad=rng.choice([0, 0, 0, 1, 2, 5]))
    if kind == "masked":
        return dict(kind=kind, prec=rng.choice(["fp64", "split"]), m=_log_int(rng, 200, 2228),
                    n=_log_int(rng, 1000, 16384), k=_log_int(rng, 200, 2228),
                    transa=rng.random() < 0.3, blk=rng.choice([48, 48, 64, 32]),
                    density=round(rng.uniform(0.1, 0.6), 3))
    if kind == "plan":
        return dict(kind=kind, prec=rng.choice(["fp64", "split"]), nao=_log_int(rng, 300, 2228),
                    nbatch=_log_int(rng, 8, 96), gmin=128, gmax=_log_int(rng, 512, 4096),
                    dmin=0.05, dmax=round(rng.uniform(0.3, 0.6), 3), nset=rng.randint(1, 3),
                    blk=64)
    if kind == "host":
        return dict(kind=kind, nao=_log_int(rng, 300, 1200), ngrid=_log_int(rng, 2000, 12000),
                    nset=rng.randint(1, 2), blk=48, density=round(rng.uniform(0.15, 0.5), 3),
                    mask="centres")
    case = dict(kind=kind, nao=_log_int(rng, 300, 4000), ngrid=_log_int(rng, 2048, 32768),
                nset=rng.randint(1, 4), blk=rng.choice([64, 64, 48]),
                density=round(rng.uniform(0.1, 0.5), 3),
                mask=rng.choice(["centres", "centres", "bernoulli"]))
    if kind == "rho":
        case["prec"] = rng.choice(["fp64", "split"])
    # no more masked work than the listed molecule's, and its tables fit beside others
    while _pairs(case) > 3 * 16384 * (0.3 * 2228) ** 2 or case["nao"] * case["ngrid"] > 4e7:
        case["ngrid"] = case["ngrid"] * 3 // 4
    return case


def _pairs(case):
    """Masked (row, column, point) products, from below (the lists' mean length)."""
    n = case["density"] * case["nao"]
    return case["nset"] * case["ngrid"] * n * n


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(shape, g):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0)


def _symmetric(nset, nao, g):
    a = _uniform((nset, nao, nao), g)
    return (0.5 * (a + a.transpose(1, 2))).contiguous()


def _points(tab, ngrid, blk):
    """(rows, blocks) tile mask -> (rows, points) bool."""
    return tab.bool().repeat_interleave(blk, dim=1)[:, :ngrid]


def _molecule(nao, rng):
    """s, p, d, f shells of nao orbitals on atom centres: (centre of shell, l, alpha, row)."""
    natom = max(2, nao // 20)
    box = 16.0 / BOHR * (natom / 110.0) ** (1.0 / 3.0)
    centres = rng.uniform(0.0, box, (natom, 3))
    ls, left = [], nao
    while left:
        l = min(int(rng.choice([0, 1, 2, 3], p=[0.05, 0.15, 0.3, 0.5])), (left - 1) // 2)
        ls.append(l)
        left -= 2 * l + 1
    l = np.array(ls)
    atom = np.sort(rng.integers(0, natom, len(l)))
    alpha = np.exp(rng.uniform(np.log(0.05), np.log(20.0), len(l)))
    row = np.concatenate([[0], np.cumsum(2 * l + 1)[:-1]])
    return centres, atom, l, alpha, row


def _orbitals(mol, ngrid, blk, density, rng):
    """phi (nao, ngrid) and its tile mask: blocks of points around the centres, the
    `density` fraction of (shell, block) tiles with the largest |phi| kept."""
    centres, atom, l, alpha, row = mol
    nblk = -(-ngrid // blk)
    at = np.repeat(rng.integers(0, len(centres), nblk), blk)[:ngrid]
    pts = centres[at] + rng.normal(0.0, 1.5, (ngrid, 3))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    p, c = dev(pts.T), dev(centres[atom])
    al = dev(alpha)
    norm = dev((2 * alpha / np.pi) ** 0.75 * (4 * alpha) ** (l / 2))
    nao = int((2 * l + 1).sum())
    ao = torch.empty(nao, ngrid, dtype=torch.float64, device="cuda")
    shmax = torch.empty(len(l), nblk, dtype=torch.float64, device="cuda")
    for q in range(4):
        sh = np.nonzero(l == q)[0]
        if not len(sh):
            continue
        s = dev(sh)
        x, y, z = (p[i][None, :] - c[s, i][:, None] for i in range(3))
        r2 = x * x + y * y + z * z
        radial = norm[s][:, None] * torch.exp(-al[s][:, None] * r2)
        if q == 0:
            poly = [torch.ones_like(x)]
        elif q == 1:
            poly = [x, y, z]
        elif q == 2:
            poly = [x * y, y * z, 3 * z * z - r2, x * z, x * x - y * y]
        else:
            poly = [y * (3 * x * x - y * y), x * y * z, y * (5 * z * z - r2),
                    z * (5 * z * z - 3 * r2), x * (5 * z * z - r2), z * (x * x - y * y),
                    x * (x * x - 3 * y * y)]
        rows = dev(row[sh])
        top = torch.zeros(len(sh), nblk * blk, dtype=torch.float64, device="cuda")
        for f, h in enumerate(poly):
            v = radial * h
            ao[rows + f] = v
            torch.maximum(top[:, :ngrid], v.abs(), out=top[:, :ngrid])
        shmax[s] = top.view(len(sh), nblk, blk).amax(2)
    keep = max(1, int(round(density * shmax.numel())))
    cut = torch.topk(shmax.flatten(), keep).values[-1]
    shell_of = dev(np.repeat(np.arange(len(l)), 2 * l + 1))
    tab = (shmax >= cut)[shell_of].to(torch.uint8).contiguous()
    ao *= _points(tab, ngrid, blk)
    return ao, tab


def _table(case, seed):
    """phi and tile mask of a rho, host or fock case."""
    if case["mask"] == "centres":
        rng = np.random.default_rng(seed)
        return _orbitals(_molecule(case["nao"], rng), case["ngrid"], case["blk"],
                         case["density"], rng)
    g = _gen(seed + 1)
    nao, ngrid, blk, shell = case["nao"], case["ngrid"], case["blk"], 8
    nblk = -(-ngrid // blk)
    on = torch.rand((-(-nao // shell), nblk), generator=g, device="cuda") < case["density"]
    tab = on.repeat_interleave(shell, dim=0)[:nao].to(torch.uint8).contiguous()
    ao = torch.randn((nao, ngrid), generator=g, device="cuda", dtype=torch.float64)
    ao *= _points(tab, ngrid, blk)
    return ao, tab


def _prec(case):
    return cm.PREC_OZAKI_INT8 if case["prec"] == "split" else cm.PREC_FP64


def _gemm_inputs(case, seed):
    g = _gen(seed)
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    a = _uniform((k, m + pad) if case["transa"] else (m, k + pad), g)
    b = _uniform((n, k + pad) if case["transb"] else (k, n + pad), g)
    return (a.float(), b.float()) if case["dtype"] == "f32" else (a, b)


def _masked_inputs(case, seed):
    g = _gen(seed)
    m, n, k, blk = case["m"], case["n"], case["k"], case["blk"]
    a = _uniform((k, m) if case["transa"] else (m, k), g)
    b = _uniform((k, n), g)
    tab = (torch.rand((k, -(-n // blk)), generator=g, device="cuda") < case["density"])
    tab = tab.to(torch.uint8)
    b *= _points(tab, n, blk)
    return a, b, tab


def _batches(case, seed):
    """The plan's batches: (phi, mask, points, matrices) of one molecule.  The sizes are the
    case's, the molecule, the points and which tiles are kept the seed's."""
    sizes, rng = np.random.default_rng(case["nbatch"]), np.random.default_rng(seed)
    mol = _molecule(case["nao"], rng)
    for _ in range(case["nbatch"]):
        ngrid = int(math.exp(sizes.uniform(math.log(case["gmin"]), math.log(case["gmax"]))))
        density = float(sizes.uniform(case["dmin"], case["dmax"]))
        nset = int(sizes.integers(1, case["nset"] + 1))
        ao, tab = _orbitals(mol, ngrid, case["blk"], density, rng)
        yield ao, tab, ngrid, nset


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "gemm":
        a, b = _gemm_inputs(case, seed)
        state.update(a=a, b=b, c=torch.zeros(case["m"], case["n"], dtype=a.dtype, device="cuda"))
    elif kind == "masked":
        a, b, tab = _masked_inputs(case, seed)
        state.update(a=a, b=b, tab=tab,
                     c=torch.zeros(case["m"], case["n"], dtype=torch.float64, device="cuda"))
    elif kind == "plan":
        made = list(_batches(case, seed))
        dms = _symmetric(case["nset"], case["nao"], _gen(seed))
        flat = torch.zeros(sum(g * s for _, _, g, s in made), dtype=torch.float64, device="cuda")
        batches, at = [], 0
        for ao, tab, ngrid, nset in made:
            rho = flat[at:at + nset * ngrid].view(nset, ngrid)
            at += nset * ngrid
            batches.append((rho, ao, ao, tab, nset))
        state.update(rho=flat, dms=dms, plan=cm.AodmPlan(batches, dms, case["blk"], _prec(case)))
    else:
        ao, tab = _table(case, seed)
        g = _gen(seed)
        nao, ngrid, nset = case["nao"], case["ngrid"], case["nset"]
        if kind == "fock":
            # quadrature weights times a potential: both signs, a few orders of magnitude
            w = torch.randn((nset, ngrid), generator=g, device="cuda", dtype=torch.float64)
            state.update(ao=ao, tab=tab, w=w * w * w, v=torch.zeros(
                nset, nao, nao, dtype=torch.float64, device="cuda"))
        else:
            rho = torch.zeros(nset, ngrid, dtype=torch.float64, device="cuda")
            state.update(ao=ao, tab=tab, dms=_symmetric(nset, nao, g), rho=rho)
            if kind == "host":
                state.update({q: state[q].cpu().numpy() for q in ("ao", "tab", "dms", "rho")})
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("gemm", "masked"):
        a, b, c = state["a"], state["b"], state["c"]
        m, n, k = case["m"], case["n"], case["k"]
        c.zero_()
        if kind == "masked":
            tab = state["tab"]
            cm.matmul_non0tab_ex(c, a, b, m, n, k, a.shape[1], b.shape[1], n, case["transa"],
                                 False, tab, tab.shape[1], case["blk"], _prec(case))
        else:
            f = cm.matmul_f32 if case["dtype"] == "f32" else cm.matmul_ex
            f(c, a, b, m, n, k, a.shape[1], b.shape[1], n, case["transa"], case["transb"],
              _prec(case))
        return c
    if kind == "plan":
        state["rho"].zero_()
        state["plan"].run()
        return state["rho"]
    ao, tab = state["ao"], state["tab"]
    nao, ngrid = ao.shape
    strides = shape = (nao, ngrid)
    if kind == "fock":
        state["v"].zero_()
        cm.aodm_fock(state["v"], state["w"], ao, ao, strides, shape, case["nset"], tab,
                     tab.shape[1], case["blk"])
        return state["v"]
    rho = state["rho"]
    if kind == "host":
        rho[:] = 0.0
        cm.aodmao2rho_anyway(rho, state["dms"], ao, ao, strides, shape, case["nset"], tab,
                             tab.shape[1])
        return rho
    rho.zero_()
    cm.aodmao2rho_ex(rho, state["dms"], ao, ao, strides, shape, case["nset"], tab, tab.shape[1],
                     case["blk"], _prec(case))
    return rho


def work(case):
    """Inputs once and outputs once.  The masks are random and their lists' mean length is
    density * nao (a lower bound of the squares' mean); phi's masked tiles are not read, and
    of a symmetric product with one phi on both sides one half is enough."""
    kind = case["kind"]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=(4 if case["dtype"] == "f32" else 8) * (m * k + k * n + m * n),
                    flops=2 * m * n * k)
    if kind == "masked":
        m, n, k, d = case["m"], case["n"], case["k"], case["density"]
        return dict(bytes=8 * (m * k + d * k * n + m * n) + k * n / case["blk"],
                    flops=2 * m * n * k * d)
    nao = case["nao"]
    if kind == "plan":
        # log-uniform sizes, uniform densities and numbers of matrices: the means
        points = case["nbatch"] * (case["gmax"] - case["gmin"]) / math.log(
            case["gmax"] / case["gmin"])
        d, sets = 0.5 * (case["dmin"] + case["dmax"]), 0.5 * (1 + case["nset"])
        return dict(bytes=8 * (points * d * nao + case["nset"] * nao * nao + sets * points),
                    flops=points * sets * (d * nao) ** 2)
    ngrid, nset, d = case["ngrid"], case["nset"], case["density"]
    return dict(bytes=8 * (d * nao * ngrid + nset * (nao * nao + ngrid)) + nao * ngrid / case["blk"],
                flops=_pairs(case))


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
def _dense_rho(ao, dms):
    return torch.stack([(ao * (d @ ao)).sum(0) for d in dms])


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        a, b = (x.double() for x in _gemm_inputs(case, seed))
        m, n, k = case["m"], case["n"], case["k"]
        a = a[:, :m].t() if case["transa"] else a[:, :k]
        b = b[:, :k].t() if case["transb"] else b[:, :n]
        return a @ b
    if kind == "masked":
        a, b, _ = _masked_inputs(case, seed)
        return (a.t() if case["transa"] else a) @ b
    if kind == "plan":
        dms = _symmetric(case["nset"], case["nao"], _gen(seed))
        return torch.cat([_dense_rho(ao, dms[:nset]).flatten()
                          for ao, _, _, nset in _batches(case, seed)])
    ao, _ = _table(case, seed)
    g = _gen(seed)
    nset, nao, ngrid = case["nset"], case["nao"], case["ngrid"]
    if kind == "fock":
        w = torch.randn((nset, ngrid), generator=g, device="cuda", dtype=torch.float64)
        return torch.stack([(ao * x) @ ao.t() for x in w * w * w])
    rho = _dense_rho(ao, _symmetric(nset, nao, g))
    return rho.cpu().numpy() if kind == "host" else rho
