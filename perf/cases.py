"""The workloads this library is timed on, through its public entry points.

Each case is one call (or the short sequence of calls) that a PNAMP or GCM program makes:
projected kernels of a few (q, q') pairs over an Euler x gauge mesh in one of the arithmetic
forms, from host buffers or from device buffers, the one- and two-body densities, the
norm-only pass of the learned mode, and a training step of its network. `listed` names the
fixed cases, `draw` makes one more of the same ranges, `prepare` makes what the program has
in hand (vacua, the context, its output buffers), `run` is one pass, `work` the least work a
pass can be done with, and `exact` the same outputs from plain torch in FP64.
"""
import math
import os

import numpy as np
import torch

from sccm_gb300.basis import NOBS, SHELLS, Mesh, ModelSpace, q2_operators
from sccm_gb300.formats import mscheme_pairs
from sccm_gb300.mlp import MLP
from sccm_gb300.pnamp import PnampContext, rho2b_tables
from sccm_gb300.synth import SHELL_NUCLEONS, deformed_vacuum, ti48_workload

NK, JJMAX = 13, 6
TRAIN_INPUTS = 25               # the learned mode's network inputs
LR = 1e-3


def _case(name, kind, shell, form, mix, mesh, npairs):
    na, nb, ng, nf = mesh
    return {"name": name, "kind": kind, "shell": shell, "form": form, "mix": mix, "nalp": na, "nbet": nb,
            "ngam": ng, "nfom": nf, "npairs": npairs}


def listed():
    return [
        # one small sd-shell pair called from the host, as an interactive check of a vacuum does:
        # 36 Euler points x 9 gauge points, dominated by launches and copies
        _case("sd_pair_small", "pair", "sd", "fp64", False, (3, 4, 3, 3), 1),
        # the sd benchmark configuration: vacua that mix protons and neutrons, plain FP64, the
        # per-pair host call that replaces the reference's subroutine
        _case("sd_pnmix_fp64", "pair", "sd", "fp64", True, (8, 16, 8, 7), 1),
        # the pf benchmark configuration (charge-conserving vacua), plain FP64, device buffers,
        # with the J/K projection
        _case("pf_fp64", "device", "pf", "fp64", False, (10, 20, 10, 9), 1),
        # the same in the headline form of bench.py, four pairs per call
        _case("pf_tc6", "device", "pf", "tc6", False, (10, 20, 10, 9), 4),
        # the same in double-float through the host-buffer batch call, as the file driver does
        _case("pf_df64_host", "batch", "pf", "df64", False, (10, 20, 10, 9), 2),
        # proton-neutron mixing pf vacua in the tensor-core form
        _case("pf_pnmix_tc6", "device", "pf", "tc6", True, (10, 20, 10, 9), 1),
        # the same vacua in double-float on a coarse mesh (the learned mode's coarse pass sizes)
        _case("pf_pnmix_df64", "device", "pf", "df64", True, (4, 8, 4, 9), 4),
        # the shipped Ti48 / KB3G vacua (proton-neutron pairing, some nearly empty levels) in FP64
        _case("ti48_fp64", "batch", "ti48", "fp64", True, (3, 6, 3, 7), 4),
        # cross-shell sd+pf, the largest model space, odd mesh sizes
        _case("sdpf_df64", "device", "sdpf", "df64", False, (5, 9, 5, 11), 1),
        # transition densities of the projected states (rho1b and rho2b in one pass)
        _case("pf_densities", "densities", "pf", "df64", False, (6, 12, 6, 9), 1),
        # the learned mode's exact norm on a fine mesh, with the per-gauge-point values
        _case("pf_norm_items", "norm_items", "pf", "df64", False, (8, 16, 8, 11), 2),
        # one step of the learned mode's network training at its batch size
        {"name": "mlp_train", "kind": "train", "rows": 16384, "width": 256, "depth": 4},
    ]


# kernel points times (n / 40)^3 that one case may hold: the largest listed case
_MOST = 6.48e5


def draw(rng):
    if rng.random() < 0.12:
        return {"kind": "train", "rows": int(math.exp(rng.uniform(math.log(1000), math.log(40000)))),
                "width": rng.choice([64, 128, 200, 256]), "depth": rng.randint(2, 5)}
    kind = rng.choice(["pair", "device", "device", "batch", "densities", "norm_items"])
    shell = rng.choice(["sd", "pf", "pf", "sdpf", "ti48"])
    form = rng.choice(["fp64", "df64", "tc6"]) if kind in ("pair", "device", "batch") else rng.choice(["fp64", "df64"])
    mix = True if shell == "ti48" else rng.random() < 0.5
    n = 40 if shell == "ti48" else _n(shell)
    most = _MOST * (0.12 if form == "fp64" else 0.4) * (0.35 if mix else 1.0)
    while True:
        c = _case("", kind, shell, form, mix, (rng.randint(2, 10), rng.randint(3, 20), rng.randint(2, 10),
                                               rng.choice([3, 4, 5, 6, 7, 8, 9, 11])),
                  1 if kind == "pair" else rng.randint(1, 4))
        pts = c["nalp"] * c["nbet"] * c["ngam"] * c["nfom"] ** 2 * c["npairs"]
        if pts * (n / 40.0) ** 3 <= most:
            break
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _n(shell):
    return 2 * sum(tj + 1 for _, _, tj in SHELLS[shell])


_spaces = {}


def _space(shell):
    """(model space, record list, quadrupole operators) of a shell: enumerations, no data."""
    if shell not in _spaces:
        sp = ModelSpace(SHELLS[shell], *SHELL_NUCLEONS[shell])
        _spaces[shell] = (sp, mscheme_pairs(sp), q2_operators(sp))
    return _spaces[shell]


def _ti48():
    if "ti48" not in _spaces:
        root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
        _spaces["ti48"] = ti48_workload(Mesh(1, 1, 1, 3), os.path.join(root, "tests", "golden", "reference_pins.npz"))
    return _spaces["ti48"]


def _mesh(c):
    return Mesh(c["nalp"], c["nbet"], c["ngam"], c["nfom"])


def _problem(c, seed):
    """(sp, e0, t1b, recs, vbar, q2, pairs): `npairs` pairs of seeded vacua and an interaction.

    Synthetic shells: deformed BCS vacua as the benchmark configurations draw them (beta2 in
    [0, 0.5], gamma in [0, 60] degrees, a random T-even rotation) and normal m-scheme matrix
    elements; ti48: pairs of the shipped vacua with the shipped KB3G interaction."""
    rng = np.random.default_rng([11, seed])
    if c["shell"] == "ti48":
        w = _ti48()
        k = [rng.integers(0, len(w.vacua), 2) for _ in range(c["npairs"])]
        return w.sp, w.e0, w.t1b, w.recs, w.vbar, w.q2, [(*w.vacua[i], *w.vacua[j]) for i, j in k]
    sp, recs, q2 = _space(c["shell"])
    spe = rng.uniform(-4.0, 0.0, len(sp.orbits))
    t1b = np.diag([spe[o] for o in sp.orbit]).astype(complex)
    vbar = 0.5 * rng.standard_normal(len(recs))

    def vac():
        return deformed_vacuum(sp, spe, rng.uniform(0.0, 0.5), rng.uniform(0.0, 60.0), rng, q2=q2, pn_mix=c["mix"])
    return sp, 0.0, t1b, recs, vbar, q2, [(*vac(), *vac()) for _ in range(c["npairs"])]


def _train_inputs(c, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    rows = c["rows"]
    x = torch.randn(rows, TRAIN_INPUTS, generator=g)
    y = torch.randn(rows, 2, generator=g) * 0.5 + x[:, :2]
    w = torch.rand(rows, generator=g) + 0.05
    dims = [TRAIN_INPUTS] + [c["width"]] * c["depth"] + [3]
    npar = sum(i * o + o for i, o in zip(dims, dims[1:]))
    # parameters and Adam moments as after some steps of training
    rng = np.random.default_rng([12, seed])
    flat = np.concatenate([np.concatenate([(rng.standard_normal(i * o) / math.sqrt(i)).astype(np.float32),
                                           (0.1 * rng.standard_normal(o)).astype(np.float32)])
                           for i, o in zip(dims, dims[1:])])
    m = torch.randn(npar, generator=g) * 1e-3
    v = torch.rand(npar, generator=g) * 1e-5 + 1e-6
    return x, y, w, dims, torch.from_numpy(flat), m, v


def prepare(case, seed):
    dev = torch.device("cuda")
    if case["kind"] == "train":
        x, y, w, _, flat, m, v = _train_inputs(case, seed)
        net = MLP(TRAIN_INPUTS, case["width"], case["depth"], 3, seed=0, device=dev)
        return {"kind": "train", "net": net, "x": x.to(dev), "y": y.to(dev), "w": w.to(dev), "flat": flat.to(dev),
                "m": m.to(dev), "v": v.to(dev)}
    sp, e0, t1b, recs, vbar, q2, pairs = _problem(case, seed)
    mesh = _mesh(case)
    ctx = PnampContext(sp, e0, t1b, recs, vbar, mesh, q2=q2, form=case["form"])
    s = {"kind": case["kind"], "ctx": ctx, "npairs": len(pairs)}
    if case["kind"] == "pair":
        s["pair"] = pairs[0]
    elif case["kind"] in ("batch", "densities"):
        s["packed"] = PnampContext.pack_pairs(pairs)
    else:
        P, G = ctx.n_euler, mesh.n_gauge
        s["uv"] = torch.from_numpy(PnampContext.pack_pairs(pairs)).to(dev)
        s["z"] = torch.zeros((len(pairs), NOBS, P, 2), dtype=torch.float64, device=dev)
        s["st"] = torch.zeros((len(pairs), P), dtype=torch.int32, device=dev)
        if case["kind"] == "device":
            s["proj"] = torch.zeros((len(pairs), 5, JJMAX + 1, NK, NK, 2), dtype=torch.float64, device=dev)
        else:
            s["g"] = torch.zeros((len(pairs), P, G, 4), dtype=torch.float64, device=dev)
            k = torch.arange(len(pairs), dtype=torch.int32, device=dev).repeat_interleave(P)
            e = torch.arange(P, dtype=torch.int32, device=dev).repeat(len(pairs))
            s["items"] = torch.stack([k, e], 1).contiguous()
    return s


def run(s):
    kind = s["kind"]
    if kind == "train":
        net = s["net"]
        net.params.copy_(s["flat"])
        net.m.copy_(s["m"])
        net.v.copy_(s["v"])
        net.step = 20
        loss = net.train_step(s["x"], s["y"], s["w"], lr=LR)
        return {"loss": loss, "out": net.acts[-1], "grads": net.grads, "params": net.params, "m": net.m, "v": net.v}
    ctx = s["ctx"]
    if kind == "pair":
        r = ctx.pair(*s["pair"])
        k = ctx.project(r.zres, chop=False)
        return {"z": r.zres, "st": r.status, "njkk": k["njkk"], "hjkk": k["hjkk"]}
    if kind == "batch":
        z, st = ctx.batch(s["packed"])
        return {"z": z, "st": st}
    if kind == "densities":
        z, st, r1, r2 = ctx.batch_densities(s["packed"])
        return {"z": z, "st": st, "rho1b": r1, "rho2b": r2}
    stream = torch.cuda.current_stream().cuda_stream
    n = s["npairs"]
    if kind == "device":
        ctx.batch_device(n, s["uv"].data_ptr(), s["z"].data_ptr(), s["st"].data_ptr(), stream)
        ctx.project_device(n, s["z"].data_ptr(), s["proj"].data_ptr(), False, stream)
        # N^J and H^J, the fields the Hill-Wheeler solve reads
        return {"z": s["z"], "st": s["st"], "proj": s["proj"][:, :2]}
    ctx.set_outputs("norm")
    ctx.batch_items_device(n, s["uv"].data_ptr(), s["items"].shape[0], s["items"].data_ptr(), s["z"].data_ptr(),
                           s["st"].data_ptr(), s["g"].data_ptr(), stream)
    ctx.set_outputs("all")
    return {"z": s["z"], "st": s["st"], "g": s["g"]}


def work(case):
    """Inputs read once, outputs written once, and the arithmetic of the smallest algorithm:
    per skew matrix of order N its inverse with the Pfaffian (N^3 / 2 complex multiply-adds)
    and two products with a real matrix (1.5 N^3 real x complex), per two-body record 12
    multiply-adds. Charge-conserving vacua need 2 NFOM matrices of order n / 2 per Euler
    point (the species separate and each depends on its own gauge angle), others NFOM^2 of
    order n."""
    if case["kind"] == "train":
        dims = [TRAIN_INPUTS] + [case["width"]] * case["depth"] + [3]
        npar = sum(i * o + o for i, o in zip(dims, dims[1:]))
        rows = case["rows"]
        mm = sum(i * o for i, o in zip(dims, dims[1:]))
        return {"bytes": 4 * (rows * (TRAIN_INPUTS + 3 + 3) + 7 * npar),
                "flops": 2.0 * rows * (3 * mm - dims[0] * dims[1])}
    n = 40 if case["shell"] == "ti48" else _n(case["shell"])
    nrec = {"sd": 2570, "pf": 14442, "ti48": 14442, "sdpf": 50508}[case["shell"]]
    P = case["nalp"] * case["nbet"] * case["ngam"]
    G = case["nfom"] ** 2
    order, mats = (n, G) if case["mix"] else (n // 2, 2 * case["nfom"])
    norm_only = case["kind"] == "norm_items"
    per = order ** 3 * (4.0 / 3.0 if norm_only else 10.0)
    rec = 0.0 if norm_only else 24.0 * nrec * (G if case["mix"] else case["nfom"])
    if case["kind"] == "densities":
        rec *= 2.0
    b = case["npairs"] * (4 * n * n * 8 + NOBS * P * 16 + P * 4)
    if case["kind"] in ("pair", "device"):
        b += case["npairs"] * 2 * 7 * NK * NK * 16
    if norm_only:
        b += case["npairs"] * P * G * 32
    return {"bytes": b, "flops": case["npairs"] * P * (mats * per + rec)}


# ------------------------------------------------------------------ the same numbers in plain torch, FP64
def _small_d(tj, beta):
    """d^j(beta) = exp(-i beta J_y), basis m = j .. -j, for every beta of a vector: [E, d, d]."""
    j = tj / 2.0
    m = j - np.arange(tj + 1)
    up = np.sqrt(j * (j + 1) - m[1:] * (m[1:] + 1))
    jp = np.diag(up, 1)
    jy = torch.from_numpy((jp - jp.T) / 2j).to(beta.device)
    w, u = torch.linalg.eigh(jy)
    ph = torch.exp(-1j * beta[:, None] * w[None, :].to(torch.complex128))
    return (u[None] * ph[:, None, :]) @ u.conj().T


def _pfaffian(A):
    """Pfaffians of skew matrices [B, N, N] by 2 x 2 elimination with row pivoting."""
    B, N = A.shape[0], A.shape[1]
    b = torch.arange(B, device=A.device)
    pf = torch.ones(B, dtype=A.dtype, device=A.device)
    while N > 2:
        q = 1 + A[:, 0, 1:].abs().argmax(1)
        r1, rq = A[b, 1].clone(), A[b, q].clone()
        A[b, 1], A[b, q] = rq, r1
        c1, cq = A[b, :, 1].clone(), A[b, :, q].clone()
        A[b, :, 1], A[b, :, q] = cq, c1
        s = A[:, 0, 1]
        pf = pf * torch.where(q == 1, s, -s)
        w, v = A[:, 0, 2:], A[:, 1, 2:] / s[:, None]
        A = A[:, 2:, 2:] + v[:, :, None] * w[:, None, :] - w[:, :, None] * v[:, None, :]
        N -= 2
    return pf * A[:, 0, 1]


class _Exact:
    def __init__(self, case, seed):
        self.sp, self.e0, t1b, recs, vbar, q2, self.pairs = _problem(case, seed)
        self.mesh = _mesh(case)
        dev = self.dev = torch.device("cuda")
        sp, n = self.sp, self.sp.nlev
        self.t1b = torch.from_numpy(np.real(t1b)).to(dev)
        self.i, self.j, self.k, self.l = (torch.from_numpy(np.asarray(recs)[:, c].astype(np.int64)).to(dev) for c in range(4))
        self.v = torch.from_numpy(np.asarray(vbar)).to(dev)
        self.d = (self.i + self.j != self.k + self.l).to(torch.float64)
        self.q2 = torch.from_numpy(np.asarray(q2)).to(dev)
        jp, jm = np.zeros((n, n)), np.zeros((n, n))
        for a in range(n):
            jj, m = sp.twoj[a] / 2.0, sp.twom[a] / 2.0
            if sp.twom[a] > -sp.twoj[a]:
                jm[a + 1, a] = math.sqrt(jj * (jj + 1) - m * (m - 1))
                jp[a, a + 1] = jm[a + 1, a]
        self.jp, self.jm = (torch.from_numpy(a).to(dev) for a in (jp, jm))
        self.mz = torch.from_numpy(sp.twom / 2.0).to(dev)
        self.jj = torch.from_numpy(sp.twoj / 2.0 * (sp.twoj / 2.0 + 1)).to(dev)
        self.euler = torch.from_numpy(self.mesh.euler_points()).to(dev)
        nf = self.mesh.nfom
        phi = torch.arange(nf, dtype=torch.float64, device=dev) * (2 * math.pi / nf)
        self.php, self.phn = phi.repeat_interleave(nf), phi.repeat(nf)
        self.gph = torch.exp(-1j * (self.php * sp.nprot + self.phn * sp.nneut))

    def rotation(self, eul):
        sp, n = self.sp, self.sp.nlev
        m = self.mz.to(torch.complex128)
        R = torch.zeros((eul.shape[0], n, n), dtype=torch.complex128, device=self.dev)
        cache = {}
        for s, d in sp.blocks():
            tj = int(sp.twoj[s])
            if tj not in cache:
                cache[tj] = _small_d(tj, eul[:, 1])
            R[:, s:s + d, s:s + d] = cache[tj]
        ea = torch.exp(-1j * eul[:, 0, None] * m[None])
        eg = torch.exp(-1j * eul[:, 2, None] * m[None])
        return ea[:, :, None] * R * eg[:, None, :]

    def chunks(self, norm_only):
        n, G = self.sp.nlev, self.mesh.n_gauge
        per = G * (16.0 * (2 * n) ** 2 * 3 + (0 if norm_only else 16.0 * len(self.v) * 6))
        return max(1, int(6e9 / per))

    def pair(self, U0, V0, U1, V1, norm_only=False, point=None):
        """ZRES [NOBS, P] and, through `point(e0, e1, N, rho, k10, k01)`, every gauge point."""
        dev, n, G = self.dev, self.sp.nlev, self.mesh.n_gauge
        U0, V0, U1, V1 = (torch.from_numpy(np.asarray(a, dtype=np.float64)).to(dev) for a in (U0, V0, U1, V1))
        h = n // 2
        Z0, W = V0 @ torch.linalg.inv(U0), V1 @ torch.linalg.inv(U1)
        eye = torch.eye(n, dtype=torch.float64, device=dev)
        det = [torch.exp(-0.25 * torch.linalg.slogdet(eye + Z.T @ Z)[1]) for Z in (Z0, W)]
        pre = det[0] * det[1] * (-1.0 if (n * (n + 1) // 2) % 2 else 1.0)
        c = torch.complex128
        ph = torch.where(torch.arange(n, device=dev)[None] < h, self.php[:, None], self.phn[:, None])
        D = torch.exp(1j * ph)                                                   # [G, n]
        P = self.euler.shape[0]
        out = torch.zeros((NOBS, P), dtype=c, device=dev)
        step = self.chunks(norm_only)
        for e0 in range(0, P, step):
            eul = self.euler[e0:e0 + step]
            E = eul.shape[0]
            R = self.rotation(eul)
            X = R @ W.to(c) @ R.transpose(1, 2)
            M = (D[None, :, :, None] * X[:, None] * D[None, :, None, :]).reshape(-1, n, n)
            S = torch.zeros((M.shape[0], 2 * n, 2 * n), dtype=c, device=dev)
            S[:, :n, :n] = 0.5 * (M - M.transpose(1, 2))
            S[:, :n, n:], S[:, n:, :n] = -eye.to(c), eye.to(c)
            S[:, n:, n:] = -0.5 * (Z0 - Z0.T).to(c)
            N = (pre * _pfaffian(S)).reshape(E, G) * self.gph[None]
            del S, M
            o = [N]
            if norm_only:
                out[0, e0:e0 + E] = N.mean(1)
                if point:
                    point(e0, e0 + E, N, None, None, None)
                continue
            A = D[None, :, :, None] * R[:, None]
            AV, AU = A @ V1.to(c), A.conj() @ U1.to(c)
            T = torch.linalg.inv(V0.T.to(c) @ AV + U0.T.to(c) @ AU)
            YV, YU = AV @ T, AU @ T
            rho, k10, k01 = YV @ V0.T.to(c), YV @ U0.T.to(c), -(YU @ V0.T.to(c))
            del A, AV, AU, T, YV, YU
            dg = torch.diagonal(rho, dim1=2, dim2=3)
            t1 = (self.t1b.T.to(c) * rho).sum((2, 3))
            o += [dg[..., :h].sum(-1), dg[..., h:].sum(-1), t1, None, None]
            i, j, k, l = self.i, self.j, self.k, self.l
            t = rho[..., k, i] * rho[..., l, j]
            t -= rho[..., l, i] * rho[..., k, j]
            t += self.d * (rho[..., i, k] * rho[..., j, l])
            t -= self.d * (rho[..., j, k] * rho[..., i, l])
            K10, K01 = k10 - k10.transpose(2, 3), k01 - k01.transpose(2, 3)
            t += 0.25 * (K01[..., i, j] * K10[..., k, l])
            t += (0.25 * self.d) * (K01[..., k, l] * K10[..., i, j])
            o.append(t1 + (t * self.v).sum(-1) + self.e0)
            del t, K10, K01
            jp, jm, jz = self.jp.to(c), self.jm.to(c), torch.diag(self.mz).to(c)
            rp, rm, rz = jp @ rho, jm @ rho, jz @ rho
            tr = lambda x: torch.diagonal(x, dim1=2, dim2=3).sum(-1)   # noqa: E731
            j2 = (dg * self.jj).sum(-1) + tr(rp) * tr(rm) + tr(rz) ** 2 - tr(rp @ rm) - tr(rz @ rz)
            for J, f in ((jp, 0.5), (jm, 0.5), (jz, 1.0)):
                j2 = j2 + f * ((J @ k10) * (k01 @ J.T)).sum((2, 3))
            o.append(j2)
            o += [(self.q2[mu, :h].to(c) * rho[..., :, :h].transpose(2, 3)).sum((2, 3)) for mu in range(5)]
            o += [(self.q2[mu, :, :h].T.to(c) * rho[..., :, :h].transpose(2, 3)).sum((2, 3)) for mu in range(5)]
            out[0, e0:e0 + E] = N.mean(1)
            for q in range(1, 18):
                if o[q] is not None:
                    out[q, e0:e0 + E] = (N * o[q]).mean(1)
            if point:
                point(e0, e0 + E, N, rho, k10, k01)
        return out

    def project(self, z):
        """N^J and H^J [2, J, K1, K2] of one pair's ZRES [NOBS, P]."""
        e = self.euler
        axial = self.mesh.nalp * self.mesh.ngam == 1
        out = torch.zeros((2, JJMAX + 1, NK, NK), dtype=torch.complex128, device=self.dev)
        for J in range(0, JJMAX + 1, 2):
            K = torch.arange(J, -J - 1, -1, dtype=torch.float64, device=self.dev).to(torch.complex128)
            d = _small_d(2 * J, e[:, 1])
            D = torch.exp(1j * e[:, 0, None] * K)[:, :, None] * d * torch.exp(1j * e[:, 2, None] * K)[:, None, :]
            wj = (2 * J + 1) / 2.0 if axial else (2 * J + 1) / (8 * math.pi ** 2)
            for f, q in ((0, 0), (1, 6)):
                blk = torch.einsum("exy,e->xy", D, wj * e[:, 3] * z[q])
                out[f, J, JJMAX - J:JJMAX + J + 1, JJMAX - J:JJMAX + J + 1] = blk.flip(0, 1)
        return out


def _exact_train(case, seed):
    x, y, w, dims, flat, m, v = _train_inputs(case, seed)
    p = flat.double().cuda().requires_grad_(True)
    x, y, w, m, v = (a.double().cuda() for a in (x, y, w, m, v))
    a, o = x, 0
    for k, (i, u) in enumerate(zip(dims, dims[1:])):
        a = a @ p[o:o + i * u].view(u, i).T + p[o + i * u:o + i * u + u]
        o += i * u + u
        if k < len(dims) - 2:
            a = torch.tanh(a)
    s = a[:, 2].clamp(-12.0, 6.0)
    loss = (w * (0.5 * ((y - a[:, :2]) ** 2).sum(1) * torch.exp(-2 * s) + 2 * s)).mean()
    g, = torch.autograd.grad(loss, p)
    b1, b2, step = 0.9, 0.999, 21
    m1, v1 = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
    new = p.detach() - LR * (m1 / (1 - b1 ** step)) / (torch.sqrt(v1 / (1 - b2 ** step)) + 1e-8)
    return {"loss": loss.detach(), "out": a.detach(), "grads": g, "params": new, "m": m1, "v": v1}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    n = 40 if case["shell"] == "ti48" else _n(case["shell"])
    pts = case["npairs"] * case["nalp"] * case["nbet"] * case["ngam"] * case["nfom"] ** 2
    if pts * (n / 40.0) ** 3 > 4.0e5:
        return None                      # over about 20 seconds
    x = _Exact(case, seed)
    kind = case["kind"]
    P, G = x.euler.shape[0], x.mesh.n_gauge
    zs, proj, r1s, r2s, gs = [], [], [], [], []
    for pr in x.pairs:
        if kind == "densities":
            sp, tab = x.sp, rho2b_tables(x.sp)
            q = [torch.from_numpy(tab["quads"][:, c]).to(x.dev) for c in range(4)]
            blocks = {}
            for a in range(sp.nlev):
                for b in range(sp.nlev):
                    if sp.t[a] == sp.t[b] and sp.lj[a] == sp.lj[b] and sp.twom[a] == sp.twom[b]:
                        blocks.setdefault((int(sp.t[a] == -1), int(sp.lj[a]), int(sp.n[a]), int(sp.n[b]),
                                           int(sp.twoj[a])), []).append((a, b))
            r1 = torch.zeros((len(blocks), P), dtype=torch.complex128, device=x.dev)
            r2 = torch.zeros(len(q[0]), dtype=torch.complex128, device=x.dev)

            def point(e0, e1, N, rho, k10, k01):
                for b, (key, ent) in enumerate(sorted(blocks.items())):
                    a, c = (torch.tensor([t[u] for t in ent], device=x.dev) for u in (0, 1))
                    r1[b, e0:e1] = (N * rho[..., a, c].sum(-1)).mean(1) / math.sqrt(key[4] + 1.0)
                i, j, k, l = q
                for e in range(e0, e1):
                    f, u, t = rho[e - e0], k10[e - e0], k01[e - e0]
                    d = f[:, k, i] * f[:, l, j] - f[:, l, i] * f[:, k, j] + t[:, i, j] * u[:, k, l]
                    r2.add_((x.euler[e, 3] / G) * (N[e - e0, :, None] * d).sum(0))
            zs.append(x.pair(*pr, point=point))
            r1s.append(r1)
            r2s.append(r2)
        elif kind == "norm_items":
            g = torch.zeros((P, G, 4), dtype=torch.float64, device=x.dev)

            def point(e0, e1, N, rho, k10, k01):
                g[e0:e1, :, 0], g[e0:e1, :, 1] = N.real, N.imag
            zs.append(x.pair(*pr, norm_only=True, point=point))
            gs.append(g)
        else:
            zs.append(x.pair(*pr))
            proj.append(x.project(zs[-1]))
    z = torch.stack(zs)
    if kind == "pair":
        return {"z": z[0].T.contiguous(), "st": None, "njkk": proj[0][0], "hjkk": proj[0][1]}
    if kind == "batch":
        return {"z": z.transpose(1, 2).contiguous(), "st": None}
    if kind == "densities":
        return {"z": z.transpose(1, 2).contiguous(), "st": None, "rho1b": torch.stack(r1s), "rho2b": torch.stack(r2s)}
    if kind == "device":
        return {"z": torch.view_as_real(z), "st": None, "proj": torch.view_as_real(torch.stack(proj))}
    return {"z": torch.view_as_real(z), "st": None, "g": torch.stack(gs)}
