"""What a user of this framework has it do, as cases that can be timed.

Every case is a restart run as the reference's users make it: the fields of one
or many SCFT instances go in from pinned host memory, a number of iterations
runs, and the fields, the densities and the per-iteration records come back.
Single solves and batches on one grid go through ``Solver`` and the C ABI's
whole-batch transfers, sweeps over uneven grids through ``Batch``.

Precision forms: "fp64" is the drop-in, "fp32" the precision form, "fp32x2" the
finishing form below the FP32 form's RMS floor. ``keep`` says in which type the
caller keeps fields and densities: the FP32 form carries single precision, so
single solves keep its results as float32; the batch and the sweep hand theirs
over to a finishing form, which takes float64.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

PKG = "stimuli-responsive-nanodroplets_gb300"
srn = importlib.import_module(PKG)
clib = importlib.import_module(PKG + "._lib")
Batch = importlib.import_module(PKG + ".batch").Batch

NF, NSP = 13, 17
SWEEP_SIZES = ((64, 64), (96, 64), (128, 96), (192, 96), (192, 128))


def _case(name, chem, grid, ns, prec, batch, iters, graph=False, keep="float64"):
    return {"name": name, "kind": "solve", "chem": chem, "nx": grid[0], "ny": grid[1], "nz": grid[2], "ns": ns,
            "prec": prec, "batch": batch, "iters": iters, "graph": graph, "keep": keep}


def listed():
    return [
        # the smallest film of the tests and the smoke run: latency and launches
        _case("film_32x16_fp64", "film", (32, 1, 16), 64, "fp64", 1, 4),
        # the symmetric diblock melt, drop-in run of one instance
        _case("bulk_64x64_fp64", "bulk2d", (64, 1, 64), 100, "fp64", 1, 8),
        # the thin-film nanodroplet as the drop-in runs it: one instance, FP64
        _case("film_192x96_fp64", "film", (192, 1, 96), 128, "fp64", 1, 6),
        # the same film in the precision form (one structure relaxed interactively)
        _case("film_192x96_fp32", "film", (192, 1, 96), 128, "fp32", 1, 12, keep="float32"),
        # a phase-diagram row in the plain form
        _case("film_192x96_fp64_b32", "film", (192, 1, 96), 128, "fp64", 32, 1, graph=True),
        # the finishing form of a handful of sweep points
        _case("film_192x96_fp32x2_b16", "film", (192, 1, 96), 128, "fp32x2", 16, 2, graph=True),
        # the headline batch: 256 thin films over a chi_AB x chi_AC grid
        _case("film_192x96_fp32_b256", "film", (192, 1, 96), 128, "fp32", 256, 4, graph=True),
        # the droplet sweep over uneven grids, one contour resolution for all points
        {"name": "sweep_64_fp32", "kind": "sweep", "points": 64, "prec": "fp32", "iters": 8, "ns": 100, "keep": "float64"},
        # a serving pool of 64^3 bulk melts in the precision form
        _case("bulk_64c_fp32_b8", "bulk3d", (64, 64, 64), 100, "fp32", 8, 3, graph=True),
        # the four-diblock 64^3 blend with noise, one drop-in solve
        _case("blend_64c_fp64", "blend", (64, 64, 64), 128, "fp64", 1, 1),
        # a box whose lengths are no power of two and three (5 in x, odd z)
        _case("film_150x75_fp32_b4", "film", (150, 1, 75), 101, "fp32", 4, 4, graph=True, keep="float32"),
        # a 3D film (MASK 1, three axes) in the finishing form
        _case("film3d_48x32x40_fp32x2", "film", (48, 32, 40), 80, "fp32x2", 1, 2, graph=True),
    ]


def _steps(c):
    """Contour steps of one instance-iteration (all chains), about."""
    ns = c["ns"]
    return {"film": 4 * ns, "bulk2d": 2 * ns, "bulk3d": 3 * ns, "blend": 10 * ns}[c["chem"]]


def draw(rng):
    """One more case: grids from 16 to 192 points per line, odd and other lengths
    among them, every precision form, batches over a factor of 64."""
    if rng.random() < 0.1:
        return {"kind": "sweep", "points": rng.choice([9, 16, 25, 36, 49]), "prec": rng.choice(["fp32", "fp32", "fp32x2"]),
                "iters": rng.randint(2, 4), "ns": rng.randint(64, 128), "keep": "float64"}
    chem = rng.choice(["film", "film", "film", "bulk2d", "bulk3d", "film3d", "blend"])

    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        how = rng.random()
        if how < 0.4:
            n = max(lo, n // 16 * 16)  # the round sizes that most boxes have
        elif how < 0.8:
            n = max(lo, n // 2 * 2)
        return n - 1 if n > 100 and n % 2 else n

    prec = rng.choice(["fp64", "fp64", "fp32", "fp32x2"])
    if chem in ("film", "bulk2d"):
        if rng.random() < 0.3:
            nx, nz = rng.choice(SWEEP_SIZES)
        else:
            nx, nz = size(24, 192), size(16, 128)
        grid, top = (nx, 1, nz), 64
    else:
        grid, top = (size(16, 64), size(16, 64), size(16, 64)), 4
    c = _case("", "film" if chem == "film3d" else chem, grid, rng.randint(40, 128), prec, 1, 1,
              graph=rng.random() < 0.7, keep="float32" if prec == "fp32" else "float64")
    del c["name"]
    cost = grid[0] * grid[1] * grid[2] * _steps(c)
    room = 192 * 96 * 512 * (24 if prec == "fp64" else 96)  # no dearer than the largest listed cases
    top = max(1, min(top, room // cost))
    c["batch"] = int(round(math.exp(rng.uniform(0.0, math.log(top)))))
    c["iters"] = max(1, min(rng.randint(1, 6), room // (cost * c["batch"])))
    return c


# ------------------------------------------------------------------- inputs
def _surface(c, b):
    """Instance b's parameters: the chemistry of the case on its grid, with chi
    spread over the batch as a phase diagram spreads it."""
    n = max(1, math.isqrt(max(c["batch"] - 1, 0)) + 1)
    fa, fc = (b // n) / max(n - 1, 1), (b % n) / max(n - 1, 1)
    ab, ac = (20.0, 40.0) if c["batch"] == 1 else (10.0 + 20.0 * fa, 20.0 + 40.0 * fc)
    cfg = srn.configs
    if c["chem"] == "film":
        s = cfg.film2d(nx=c["nx"], nz=c["nz"], ns=c["ns"], chi_ab=ab, chi_ac=ac)
    elif c["chem"] == "bulk2d":
        s = cfg.bulk2d(nx=c["nx"], nz=c["nz"])
        s.set_chi("A", "B", ab)
    elif c["chem"] == "bulk3d":
        s = cfg.bulk3d_point(ab, ac, cfg.PLANES[b % 3], ns=c["ns"])
    else:
        s = cfg.blend3d(ns=c["ns"], seed=2 + b)
    s.NS = c["ns"]
    if c["ny"] > 1:
        s.LX, s.LY, s.LZ = (c[k] * s.DR_TARGET for k in ("nx", "ny", "nz"))
    return s


def _inputs(c, seed):
    """[(surface, w14, mask3 or None)] of a case, from the seed."""
    cfg = srn.configs
    if c["kind"] == "sweep":
        n = math.isqrt(c["points"])
        ss = cfg.sweep_surfaces(n, seed=3, sizes=SWEEP_SIZES, ns_range=(c["ns"], c["ns"]))
    else:
        ss = [_surface(c, b) for b in range(c["batch"])]
    out = []
    for b, s in enumerate(ss):
        if s.MASK:
            r = min(6.0, 0.3 * s.LX, 0.6 * s.LZ)
            out.append((s, cfg.droplet_fields(s, seed=1000 * seed + b, radius=r), cfg.substrate_mask(s)))
        else:
            fields = tuple(range(9)) if s.VOL_DBK[1] > 0 else (0, 1, 2) if s.VOL_HOMO[2] > 0 else (0, 1)
            out.append((s, cfg.uniform_fields(s.grid(), seed=1000 * seed + b, amp=0.1, fields=fields), None))
    return out


def _rng_state(b):
    return (11 + b, 22, 33)


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    inst = _inputs(case, seed)
    st = {"case": case, "noisy": any(s.DT_NOISE for s, _, _ in inst)}
    if case["kind"] == "sweep":
        b = Batch([s for s, _, _ in inst], precision=case["prec"])
        for i, (_, w, m) in enumerate(inst):
            b.set_masks(i, m)
            b.set_iteration(i, 1)
            b.set_rng(i, _rng_state(i))
        place = [b.locate(i) for i in range(b.n)]
        groups = []
        for g in range(b.groups):
            mine = sorted((slot, i) for i, (gg, slot) in enumerate(place) if gg == g)
            w_in = _pinned(len(mine), 14, b.M[mine[0][1]])
            for slot, i in mine:
                w_in[slot] = torch.from_numpy(inst[i][1])
            groups.append((clib.lib().scft_batch_context(b._h, g), w_in, _pinned(*w_in.shape), _pinned(*w_in.shape)))
        st.update(batch=b, groups=groups)
        return st
    sv = srn.Solver([s for s, _, _ in inst], precision=case["prec"], use_graph=case["graph"],
                    noise="device" if st["noisy"] else "host")
    for i, (_, w, m) in enumerate(inst):
        if m is not None:
            sv.set_masks(m, i)
        sv.set_iteration(1, i)
        sv.set_rng(_rng_state(i), i)
    w_in = _pinned(len(inst), 14, sv.M)
    for i, (_, w, _) in enumerate(inst):
        w_in[i] = torch.from_numpy(w)
    st.update(solver=sv, w_in=w_in, w=_pinned(*w_in.shape), phi=_pinned(*w_in.shape))
    return st


def run(state):
    c, lib = state["case"], clib.lib()
    keep = torch.float32 if c["keep"] == "float32" else torch.float64
    if c["kind"] == "sweep":
        for h, w_in, _, _ in state["groups"]:
            clib.check(lib.scft_set_fields_all(h, _ptr(w_in)), "scft_set_fields_all")
        res = state["batch"].run(c["iters"], chunk=c["iters"])
        out = {"rec": np.array([(r.free_energy, r.rms) for r in res])}
        for g, (h, _, w, phi) in enumerate(state["groups"]):
            clib.check(lib.scft_get_fields_all(h, _ptr(w)), "scft_get_fields_all")
            clib.check(lib.scft_get_densities_all(h, _ptr(phi)), "scft_get_densities_all")
            out["w%d" % g], out["phi%d" % g] = w.to(keep), phi.to(keep)
        return out
    sv, w, phi = state["solver"], state["w"], state["phi"]
    clib.check(lib.scft_set_fields_all(sv._h, _ptr(state["w_in"])), "scft_set_fields_all")
    if state["noisy"]:
        for i in range(sv.B):
            sv.set_iteration(1, i)
            sv.set_rng(_rng_state(i), i)
    recs = sv.iterate(c["iters"])
    clib.check(lib.scft_get_fields_all(sv._h, _ptr(w)), "scft_get_fields_all")
    clib.check(lib.scft_get_densities_all(sv._h, _ptr(phi)), "scft_get_densities_all")
    rec = np.array([[(r.free_energy, r.rms, *r.q) for r in row] for row in recs])
    return {"w": w.to(keep), "phi": phi.to(keep), "rec": rec.astype(c["keep"])}


# --------------------------------------------------------------------- work
def _species(s):
    """(kind, index, length, X-block length, fields) of every species present,
    with the reference's contour counts."""
    out = []
    for h in range(10):
        if s.VOL_HOMO[h] > 0:
            n = math.floor(s.LEN_HOMO[h] * s.NS)
            n -= 1 if n % 2 == 0 or n > s.NS else 0
            out.append(("homo", h, n, n, h, h))
    for d in range(4):
        if s.VOL_DBK[d] > 0:
            n = math.floor(s.LEN_DBK[d] * s.NS)
            n -= n % 2 == 0
            x = math.floor(s.F_INPUT_DBK[d] * n) + 1
            x -= x % 2 == 0
            fx = 0 if d == 0 else 2 * d + 1
            out.append(("dbk", d, n, x, fx, fx + 1))
    if s.MASK:
        for k in range(3):
            if s.VOL_S[k] > 0:
                n = math.floor(s.LEN_S[k] * s.NS)
                n -= n % 2 == 0
                out.append(("brush", k, n, n, 10 + k, 10 + k))
    return out


def work(case):
    """Bytes: fields in, fields and densities out, and every propagator slice
    written once and read once for the densities, at the form's width (no GPU
    holds an instance's slices on chip). Flops: two real transforms per axis and
    the factors, 5 log2 n + 3 per point and step, and the Simpson products."""
    if case["kind"] == "sweep":
        n = math.isqrt(case["points"])
        ss = srn.configs.sweep_surfaces(n, seed=3, sizes=SWEEP_SIZES, ns_range=(case["ns"], case["ns"]))
    else:
        ss = [_surface(case, b) for b in range(case["batch"])]
    width = 4 if case["prec"] == "fp32" else 8
    nbytes = flops = 0.0
    for s in ss:
        nx, ny, nz = s.grid()
        m = nx * ny * nz
        slices = sum(n * (1 if k == "homo" else 2) for k, _, n, _, _, _ in _species(s))
        per = 3 + sum(5 * math.log2(n) for n in (nx, ny, nz) if n > 1)
        nbytes += 8 * 42 * m + case["iters"] * 2 * width * m * slices
        flops += case["iters"] * m * slices * (per + 2)
    return {"bytes": nbytes, "flops": flops}


# -------------------------------------------------------------------- exact
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)


def _operator(n, alpha, wall):
    """exp(alpha d2/dx2) on one axis as a matrix: periodic, or between two walls
    (odd extension of length 2 (n + 1)), with the reference's wave numbers."""
    i = np.arange(n)
    if wall:
        m = np.arange(1, n + 1)
        S = np.sin(math.pi * np.outer(i + 1, m) / (n + 1))
        return _t((S * np.exp(-alpha * (math.pi * m / (n + 1)) ** 2)) @ S.T * (2.0 / (n + 1)))
    k = 2.0 * math.pi * (n / 2.0 - np.abs(i - n / 2.0)) / n
    c = np.cos(2.0 * math.pi * (np.outer(i, i) % n) / n) @ np.exp(-alpha * k * k) / n
    return _t(c[(i[:, None] - i[None, :]) % n])


def _drand48(state, count):
    """The next `count` values of drand48 from the 48-bit state, and all states."""
    A, C, MASK = 0x5DEECE66D, 0xB, (1 << 48) - 1
    x = np.empty(count, dtype=np.uint64)
    x[0] = (A * state + C) & MASK
    a, c, have = A, C, 1
    while have < count:
        take = min(have, count - have)
        x[have:have + take] = (x[:take] * np.uint64(a) + np.uint64(c)) & np.uint64(MASK)
        c, a, have = (a * c + c) & MASK, (a * a) & MASK, have + take
    return x


def _noise(state, count):
    """`count` Gaussians of the polar method, one per accepted pair; new state."""
    x = _drand48(state, 2 * int(count * 1.3 + 4096))
    u = 2.0 * (x.astype(np.float64) / float(1 << 48)) - 1.0
    w = u[0::2] ** 2 + u[1::2] ** 2
    ok = np.nonzero(w < 1.0)[0][:count]
    w = w[ok]
    return u[0::2][ok] * np.sqrt(-2.0 * np.log(w) / w), int(x[2 * ok[-1] + 1])


def _scft(ss, w14, mask3, iters, first_iter, rng):
    """The field iteration for instances of one grid and one set of contour
    lengths, in 64 bits: (w [B,14,M], phi [B,14,M], F [n][B], rms, Q [n][B][17])."""
    s0 = ss[0]
    nx, ny, nz = s0.grid()
    B, M, ds = len(ss), nx * ny * nz, 1.0 / (s0.NS - 1)
    L = (s0.LX, s0.LY, s0.LZ)
    dims = (nx, ny, nz)
    K = [_operator(n, ds / (L[a] / n) ** 2, bool(s0.MASK) and a == 2) if n > 1 else None for a, n in enumerate(dims)]
    spec = _species(s0)
    coat = sum(s0.VOL_S) if s0.MASK else 0.0
    act = [f for f in range(NF) if (f < 10 and s0.VOL_HOMO[f] > 0) or (f >= 10 and s0.VOL_S[f - 10] > 0)
           or any(k == "dbk" and f in (fx, fy) for k, _, _, _, fx, fy in spec)]
    avg = np.zeros(NF)
    for d in range(4):
        fx = 0 if d == 0 else 2 * d + 1
        avg[fx] += s0.F_INPUT_DBK[d] * s0.VOL_DBK[d]
        avg[fx + 1] += (1.0 - s0.F_INPUT_DBK[d]) * s0.VOL_DBK[d]
    avg[:10] += s0.VOL_HOMO
    chi = np.array([s.chi_table() for s in ss])
    live = [abs(a) > 1e-6 for a in avg[:10]] + [bool(s0.MASK) and abs(v) > 1e-6 for v in s0.VOL_S]
    chi *= np.outer(live, live)[None]
    if s0.MASK:
        avg[10:] = np.where(live[10:], s0.VOL_S, 0.0)
        avg[:10] *= 1.0 - coat
    chi, avg = _t(chi), _t(avg)
    w, p = _t(w14)[:, :NF].clone(), _t(w14)[:, NF].clone()
    phi = torch.zeros(B, NF, M, dtype=torch.float64, device=DEV)
    mask = _t(mask3) if s0.MASK else None
    recs = []

    def step(q, b):
        q = (q * b).view(B, nx, ny, nz)
        if K[2] is not None:
            q = torch.matmul(q.reshape(B, nx * ny, nz), K[2]).view(B, nx, ny, nz)
        if K[1] is not None:
            q = torch.matmul(K[1], q)
        if K[0] is not None:
            q = torch.matmul(K[0], q.reshape(B, nx, ny * nz))
        return q.reshape(B, M) * b

    def chain(q, n, switch, f0, f1):
        b0, b1 = torch.exp(ds * (-w[:, f0] / 2.0)), torch.exp(ds * (-w[:, f1] / 2.0))
        out = [q]
        for t in range(n - 1):
            out.append(step(out[-1], b0 if t < switch else b1))
        return out

    def simpson(qf, qb, lo, hi, n, Q):
        acc = qf[lo] * qb[n - 1 - lo] + qf[hi] * qb[n - 1 - hi]
        for t in range(lo + 1, hi, 2):
            acc += 4.0 * qf[t] * qb[n - 1 - t]
        for t in range(lo + 2, hi - 1, 2):
            acc += 2.0 * qf[t] * qb[n - 1 - t]
        return acc / 3.0 * ((1.0 / (n - 1)) / Q)[:, None]

    for it in range(first_iter + 1, first_iter + 1 + iters):
        phi.zero_()
        Qs = torch.zeros(B, NSP, dtype=torch.float64, device=DEV)
        lnq = torch.zeros(B, dtype=torch.float64, device=DEV)
        one = torch.ones(B, M, dtype=torch.float64, device=DEV)
        for kind, i, n, x, fx, fy in spec:
            if kind == "homo":
                qf = qb = qq = chain(one, n, n, fx, fx)
                vol, row = s0.VOL_HOMO[i] * (1.0 - coat), 4 + i
            elif kind == "dbk":
                qf, qb = chain(one, n, x - 1, fx, fy), chain(one, n, n - x, fy, fx)
                qq = qb if i < 2 else qf
                vol, row = s0.VOL_DBK[i] * (1.0 - coat), i
            else:
                qf, qb = chain(mask[:, i], n, n, fx, fx), chain(one, n, n, fx, fx)
                qq, vol, row = qf, s0.VOL_S[i], 14 + i
            Q = qq[-1].mean(1)
            Qs[:, row] = Q
            lnq += vol / ((n - 1) * ds) * torch.log(Q)
            if kind == "dbk":
                phi[:, fx] += vol * simpson(qf, qb, 0, x - 1, n, Q)
                phi[:, fy] += vol * simpson(qf, qb, x - 1, n - 1, n, Q)
            else:
                phi[:, fx] += vol * simpson(qf, qb, 0, n - 1, n, Q)
            del qf, qb, qq
        tot = phi[:, :10].sum(1) + (phi[:, 10:].sum(1) if s0.MASK else 0.0)
        H = 0.5 * (phi * torch.bmm(chi, phi)).sum(1) - (w * phi).sum(1) - p * (1.0 - phi.sum(1))
        F = H.mean(1) - lnq
        r = phi[:, act] - avg[act][None, :, None]
        ca = chi[:, act][:, :, act]
        dw = -w[:, act] + p[:, None] + torch.bmm(ca, r)
        corr = 0.5 * ca.sum((1, 2))[:, None] * r.sum(1) - (ca.sum(2)[:, :, None] * r).sum(1) if len(act) > 1 else 0.0
        g1 = s0.G1
        wn = w[:, act] + (g1 / 6.0) * dw.sum(1, keepdim=True) + (g1 - g1 / 6.0) * dw
        if s0.DT_NOISE and it <= s0.RELAXATION:
            for b in range(B):
                g, rng[b] = _noise(rng[b], M * len(act))
                # drawn point by point with x fastest, the fields of a point together
                wn[b] += s0.DT_NOISE * _t(g).view(nz, ny, nx, len(act)).permute(3, 2, 1, 0).reshape(len(act), M)
        w[:, act] = wn
        p = (wn.sum(1) + corr) / len(act)
        p = p - p.mean(1, keepdim=True)
        recs.append(torch.cat([F[:, None], ((tot - 1.0) ** 2).mean(1).sqrt()[:, None], Qs], 1))
    return torch.cat([w, p[:, None]], 1).cpu(), torch.cat([phi, tot[:, None]], 1).cpu(), torch.stack(recs).cpu()


def exact(case, seed):
    """The same restart run in 64 bits with dense operators, in torch alone."""
    inst = _inputs(case, seed)

    def go(idx):
        ss = [inst[i][0] for i in idx]
        seeds = [(33 << 32) | (22 << 16) | (11 + i) for i in idx]
        m = np.stack([inst[i][2] for i in idx]) if ss[0].MASK else None
        return _scft(ss, np.stack([inst[i][1] for i in idx]), m, case["iters"], 1, seeds)

    if case["kind"] == "sweep":
        out = {"rec": np.zeros((len(inst), 2))}
        for g, grid in enumerate(dict.fromkeys(s.grid() for s, _, _ in inst)):
            mine = [i for i, (s, _, _) in enumerate(inst) if s.grid() == grid]
            out["w%d" % g], out["phi%d" % g], rec = go(mine)
            out["rec"][mine] = rec[-1, :, :2].numpy()
        return out
    n = len(inst)
    part = max(1, min(n, 32 * 192 * 96 // (case["nx"] * case["ny"] * case["nz"])))
    done = [go(list(range(lo, min(n, lo + part)))) for lo in range(0, n, part)]
    return {"w": torch.cat([d[0] for d in done]), "phi": torch.cat([d[1] for d in done]),
            "rec": torch.cat([d[2] for d in done], 1)}
