"""Points of pairs with well conditioned U0 and V1 (sccm_gb300/csrc/point_reduced.cuh): densities
and norm from one skew inverse, and the species factorisation of charge-conserving pairs.

CPU: the identities against the oracle's literal sequence. GPU: every observable against the
oracle where the kernels can go wrong, that is matrix orders of all thread-group plans (h = 8,
12, 20, 32; n = 16, 24, 40), odd and even NFOM, Euler counts around the batch of a species-split
launch, and item lists with runs of several pairs, repeats and skipped entries.

Tolerances: identities in FP64, condition numbers of these matrices below 1e3: 1e-11. GPU against
oracle as in test_gpu_parity.py: 1e-10 for the norm, 1e-9 for the rest.
"""
import ctypes as C

import numpy as np
import pytest

from sccm_gb300.basis import NOBS, SHELLS, Mesh, ModelSpace
from sccm_gb300.synth import deformed_vacuum, make_workload
from oracle.pnamp_oracle import (Hamiltonian, gauge_matrix, kernel_triaxial, pfaf_over, rokappa, rotation_mat,
                                 uvphiomega, zbareover, zpfaffian)


def vacua(shell, mix, seed):
    sp = ModelSpace(SHELLS[shell], 2, 2)
    rng = np.random.default_rng(seed)
    spe = rng.uniform(-4.0, 0.0, len(sp.orbits))
    return sp, [deformed_vacuum(sp, spe, b, 25.0, rng, pn_mix=mix) for b in (0.1, 0.4)]


@pytest.mark.parametrize("shell,mix", [("sd", True), ("sd", False), ("pf", True)])
def test_densities_and_norm_from_one_skew_inverse(shell, mix):
    sp, ((U0, V0), (U1, V1)) = vacua(shell, mix, 5)
    h = sp.nlev // 2
    Z0, W, Wi = V0 @ np.linalg.inv(U0), V1 @ np.linalg.inv(U1), U1 @ np.linalg.inv(V1)
    R = rotation_mat(sp, 0.4, 1.3, 2.2)
    phi = (0.9, 2.6)
    A = gauge_matrix(R, *phi)
    D = np.exp(1j * np.where(np.arange(sp.nlev) < h, *phi))
    K = R.conj() @ Wi @ R.conj().T - D[:, None] * Z0 * D[None, :]
    k10 = D[:, None] * np.linalg.inv(K) * D[None, :]
    rho = -k10 @ Z0
    k01 = Z0 + Z0 @ k10 @ Z0
    for a, b in zip((rho, k10, k01), rokappa(A, U0, V0, U1, V1)):
        assert np.abs(a - b).max() <= 1e-11
    full = pfaf_over(zbareover(V0, U0)[0], *uvphiomega(A, U1, V1))[0]
    fact = zpfaffian(W)[0] * zpfaffian(K)[0]
    assert abs(full - fact) <= 1e-11 * abs(full)
    if not mix:   # each species' block depends on its own gauge angle
        for s, f in ((slice(0, h), phi[0]), (slice(h, None), phi[1])):
            Ks = (R.conj() @ Wi @ R.conj().T)[s, s] - np.exp(2j * f) * Z0[s, s]
            assert np.abs(Ks - K[s, s]).max() <= 1e-13


def check(z, ref):
    for io in range(NOBS):
        sc = np.abs(ref[:, io]).max()
        tol = 1e-10 if io == 0 else 1e-9
        assert np.abs(z[:, io] - ref[:, io]).max() <= tol * sc, io


def context(w, form):
    from sccm_gb300.pnamp import PnampContext
    return PnampContext(w.sp, w.e0, w.t1b, w.recs, w.vbar, w.mesh, q2=w.q2, form=form)


def oracle(w, i, j):
    return kernel_triaxial(w.sp, Hamiltonian(w.e0, w.t1b, w.recs, w.vbar, w.q2, w.jops), w.mesh, *w.vacua[i], *w.vacua[j])


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
@pytest.mark.parametrize("shell,mix,mesh", [("p2", False, (1, 5, 1, 4)), ("p2", True, (2, 3, 1, 3)),
                                            ("sd", False, (3, 3, 1, 2)), ("sd", True, (1, 3, 2, 4)),
                                            ("pf", False, (1, 17, 1, 5)), ("pf", True, (1, 2, 1, 3)),
                                            ("sdpf", False, (1, 5, 1, 3))])
def test_orders_and_meshes(shell, mix, mesh, form):
    w = make_workload(shell, 2, Mesh(*mesh), seed=31, pn_mix=mix)
    with context(w, form) as ctx:
        z, st = ctx.batch([(*w.vacua[0], *w.vacua[1])])
    assert st.max() == 0
    check(z[0], oracle(w, 0, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
def test_item_lists_over_split_and_mixing_pairs(form):
    """Runs of one pair, a repeat, skipped entries and pairs of both kinds in one list; the norm
    with per-gauge values as the sum over gauge points."""
    import torch
    ws = [make_workload("sd", 2, Mesh(3, 4, 3, 3), seed=31, pn_mix=m) for m in (False, True)]
    w = ws[0]
    pairs = [(*a.vacua[0], *a.vacua[1]) for a in (ws[0], ws[1], ws[0])]
    rng = np.random.default_rng(2)
    items = [(0, e) for e in range(11)] + [(1, 4), (5, 0), (2, 7), (2, 8), (0, 35), (0, 35), (-1, 3), (2, 36), (1, 0)]
    items += [(int(rng.integers(0, 3)), int(rng.integers(0, 36))) for _ in range(9)]
    good = {(p, e) for p, e in items if 0 <= p < 3 and 0 <= e < 36}
    with context(w, form) as ctx:
        P, G = ctx.n_euler, 9
        full, _ = ctx.batch(pairs)
        uv = torch.from_numpy(ctx.pack_pairs(pairs)).cuda()
        it = torch.tensor(items, dtype=torch.int32, device="cuda")
        for outputs in ("all", "norm"):
            z = torch.full((3, NOBS, P, 2), 7.0, dtype=torch.float64, device="cuda")
            st = torch.full((3, P), 99, dtype=torch.int32, device="cuda")
            g = torch.zeros((3, P, G, 4), dtype=torch.float64, device="cuda")
            ctx.set_outputs(outputs)
            ctx.batch_items_device(3, uv.data_ptr(), len(items), it.data_ptr(), z.data_ptr(), st.data_ptr(),
                                   g.data_ptr() if outputs == "norm" else 0, torch.cuda.current_stream().cuda_stream)
            ctx.set_outputs("all")
            torch.cuda.synchronize()
            zc = torch.view_as_complex(z).cpu().numpy().transpose(0, 2, 1)
            for p in range(3):
                for e in range(P):
                    if (p, e) not in good:
                        assert st[p, e] == 99 and np.all(zc[p, e] == 7 + 7j)
                        continue
                    assert st[p, e] == 0
                    cols = range(NOBS) if outputs == "all" else [0]
                    for io in cols:
                        sc = np.abs(full[p, :, io]).max()
                        assert abs(zc[p, e, io] - full[p, e, io]) <= (1e-12 if form == "fp64" else 1e-11) * sc, (p, e, io)
                    if outputs == "norm":
                        n = torch.view_as_complex(g[p, e, :, 0:2].contiguous()).mean().item()
                        assert abs(n - zc[p, e, 0]) <= 1e-13 * np.abs(full[p, :, 0]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
def test_gauge_values_of_a_split_pair_agree_with_its_factorised_sums(form):
    """A launch with H/N of every gauge point takes the n x n path for a charge-conserving pair;
    its sums are those of the species factorisation."""
    import torch
    w = make_workload("pf", 2, Mesh(1, 3, 2, 4), seed=33)
    with context(w, form) as ctx:
        P, G = ctx.n_euler, 16
        full, _ = ctx.batch([(*w.vacua[0], *w.vacua[1])])
        uv = torch.from_numpy(ctx.pack_pairs([(*w.vacua[0], *w.vacua[1])])).cuda()
        it = torch.tensor([(0, e) for e in range(P)], dtype=torch.int32, device="cuda")
        z = torch.zeros((1, NOBS, P, 2), dtype=torch.float64, device="cuda")
        st = torch.zeros((1, P), dtype=torch.int32, device="cuda")
        g = torch.zeros((1, P, G, 4), dtype=torch.float64, device="cuda")
        ctx.batch_items_device(1, uv.data_ptr(), P, it.data_ptr(), z.data_ptr(), st.data_ptr(), g.data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    zc = torch.view_as_complex(z).cpu().numpy()[0].T
    check(zc, full[0])
    N, H = (torch.view_as_complex(g[0, :, :, k:k + 2].contiguous()).cpu().numpy() for k in (0, 2))
    assert np.abs((N * H).mean(1) - full[0, :, 6]).max() <= 1e-9 * np.abs(full[0, :, 6]).max()
