"""The classes of pairs (pair_kind in sccm_gb300/csrc/point_kernels.cuh) over the range of Pfaffian scales,
gaps and fillings.

Tolerances, as in test_reduced_points.py: 1e-10 of the largest value for the norm, 1e-9 for the
other observables, in both arithmetic forms.
"""
import numpy as np
import pytest

from sccm_gb300.basis import NOBS, SHELLS, Mesh, ModelSpace, q2_operators
from sccm_gb300.formats import mscheme_pairs
from sccm_gb300.synth import deformed_vacuum


def problem(shell, nucleons, gap, seed, mix=False, nvac=2):
    """(context arguments, vacua) of seeded vacua and normal m-scheme matrix elements."""
    sp = ModelSpace(SHELLS[shell], *nucleons)
    rng = np.random.default_rng(seed)
    spe = rng.uniform(-4.0, 0.0, len(sp.orbits))
    t1b = np.diag([spe[o] for o in sp.orbit]).astype(complex)
    recs, q2 = mscheme_pairs(sp), q2_operators(sp)
    vac = [deformed_vacuum(sp, spe, 0.1 + 0.3 * k, 25.0, rng, q2=q2, gap=gap, pn_mix=mix) for k in range(nvac)]
    return (sp, 0.0, t1b, recs, 0.5 * rng.standard_normal(len(recs))), q2, vac


def check(z, ref):
    for io in range(NOBS):
        sc = np.abs(ref[:, io]).max()
        tol = 1e-10 if io == 0 else 1e-9
        assert np.abs(z[:, io] - ref[:, io]).max() <= tol * sc, io


@pytest.mark.gpu
@pytest.mark.parametrize("shell,nucleons,gap,scales", [
    ("sd", (2, 2), None, (-4, 3)), ("pf", (4, 4), None, (-3, -2, 1, 2)), ("sdpf", (4, 4), None, (-3, 1, 2)),
    ("sdpf", (2, 2), 0.5, (0, -2, 2))])
def test_results_do_not_depend_on_the_pfaffian_scale(shell, nucleons, gap, scales):
    """Cscale = 10^k with the vacuum factor iscale = k leaves every observable as it is, although the
    Pfaffians of an sd+pf pair then span 1e-192 to 1e128; at k = 0 and gap 0.5 MeV the product of
    the two species' sums is 1e39 by itself."""
    from sccm_gb300.pnamp import PnampContext
    args, q2, vac = problem(shell, nucleons, gap, 3)
    pair = [(*vac[0], *vac[1])]
    mesh = Mesh(1, 5, 2, 3)
    with PnampContext(*args, mesh, q2=q2) as ctx:
        ref, st = ctx.batch(pair)
        assert st.max() == 0
    for k in scales:
        for form in ("fp64", "df64"):
            with PnampContext(*args, mesh, q2=q2, cscale=10.0 ** k, iscale=k, form=form) as ctx:
                z, st = ctx.batch(pair)
            assert st.max() == 0, (k, form)
            check(z[0], ref[0])


# charge-conserving pairs whose V0 is well conditioned and whose V1 has nearly empty levels: outside
# the class of the single skew inverse, so their problems go by T22, one per species and gauge angle
WEAK = {"p2": ((2, 2), 0.1), "sd": ((2, 2), 0.2), "pf": ((4, 4), 0.2), "sdpf": ((4, 4), 0.3)}


def oracle(args, q2, mesh, pair, **kw):
    from oracle.pnamp_oracle import Hamiltonian, kernel_triaxial
    from sccm_gb300.basis import j_operators
    sp, e0, t1b, recs, vbar = args
    return kernel_triaxial(sp, Hamiltonian(e0, t1b, recs, vbar, q2, j_operators(sp)), mesh, *pair, **kw)


@pytest.mark.parametrize("shell", sorted(WEAK))
def test_weak_pairs_are_outside_the_reduced_class(shell):
    _, _, (b, k) = problem(shell, *WEAK[shell], 0)
    assert np.abs(k[0] @ np.linalg.inv(k[1])).max() > 40.0      # W^-1 = U1 V1^-1
    assert np.linalg.cond(b[1]) < 1e2                           # V0
    h = b[0].shape[0] // 2
    assert max(np.abs(M[:h, h:]).max() for M in (*b, *k)) == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
@pytest.mark.parametrize("shell,mesh", [("p2", (2, 3, 1, 4)), ("sd", (3, 3, 1, 3)), ("pf", (1, 5, 1, 3)),
                                        ("sdpf", (1, 3, 1, 2)), ("sd", (2, 2, 2, 1))])
def test_weak_pairs_match_the_oracle(shell, mesh, form):
    """Plain launches, densities, and the values of every gauge point, H/N or the norm alone."""
    import torch
    from oracle.pnamp_oracle import rho1b_table
    from sccm_gb300.pnamp import PnampContext
    args, q2, vac = problem(shell, *WEAK[shell], 0)
    mesh, pair = Mesh(*mesh), (*vac[0], *vac[1])
    with PnampContext(*args, mesh, q2=q2, form=form) as ctx:
        z, st = ctx.batch([pair, pair])
        zd, _, r1, r2 = ctx.batch_densities([pair])
        P, G = ctx.n_euler, mesh.n_gauge
        quads = ctx.rho2b_tables()["quads"]
        uv = torch.from_numpy(ctx.pack_pairs([pair])).cuda()
        it = torch.tensor([(0, e) for e in range(P)] + [(1, 0), (0, P)], dtype=torch.int32, device="cuda")
        zi = {}
        for outputs in ("all", "norm"):
            za = torch.zeros((1, NOBS, P, 2), dtype=torch.float64, device="cuda")
            sa = torch.zeros((1, P), dtype=torch.int32, device="cuda")
            g = torch.zeros((1, P, G, 4), dtype=torch.float64, device="cuda")
            ctx.set_outputs(outputs)
            ctx.batch_items_device(1, uv.data_ptr(), P + 2, it.data_ptr(), za.data_ptr(), sa.data_ptr(), g.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert sa.max() == 0
            zi[outputs] = torch.view_as_complex(za).cpu().numpy()[0].T, torch.view_as_complex(g.view(P, G, 2, 2)).cpu().numpy()
        ctx.set_outputs("all")
    ref, o1, o2 = oracle(args, q2, mesh, pair, rho1b=rho1b_table(args[0]), rho2b=quads)
    assert st.max() == 0
    check(z[0], ref)
    check(z[1], ref)
    check(zd[0], ref)
    assert np.abs(r1[0].T - o1).max() <= 1e-9 * np.abs(o1).max()
    o2 = mesh.euler_points()[:, 3] @ o2
    assert np.abs(r2[0] - o2).max() <= 1e-9 * np.abs(o2).max()
    check(zi["all"][0], ref)
    N, H = (zi["all"][1][:, :, k] for k in (0, 1))
    assert np.abs((N * H).mean(1) - ref[:, 6]).max() <= 1e-9 * np.abs(ref[:, 6]).max()
    assert np.abs(zi["norm"][0][:, 0] - ref[:, 0]).max() <= 1e-10 * np.abs(ref[:, 0]).max()
    assert np.abs(zi["norm"][1][:, :, 0].mean(1) - ref[:, 0]).max() <= 1e-10 * np.abs(ref[:, 0]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
@pytest.mark.parametrize("shell,mix", [("p2", False), ("p2", True), ("sd", True), ("pf", False), ("pf", True)])
def test_a_single_gauge_point_takes_the_onishi_norm(shell, mix, form):
    """NFOM = 1 of pairs in the class of the single skew inverse."""
    from sccm_gb300.pnamp import PnampContext
    args, q2, vac = problem(shell, (2, 2), None, 6, mix=mix)
    mesh, pair = Mesh(2, 2, 1, 1), (*vac[0], *vac[1])
    with PnampContext(*args, mesh, q2=q2, form=form) as ctx:
        z, st = ctx.batch([pair])
    assert st.max() == 0
    check(z[0], oracle(args, q2, mesh, pair))


@pytest.mark.gpu
@pytest.mark.parametrize("shell,nucleons", [("p2", (2, 2)), ("sd", (4, 2)), ("pf", (4, 4))])
def test_weak_and_other_pairs_of_one_batch_in_the_tensor_core_form(shell, nucleons):
    """A launch with pairs of several classes, against double-float (energies of BF16x6 within 1e-6, all
    else to rounding)."""
    from sccm_gb300.pnamp import PnampContext
    args, q2, vac = problem(shell, nucleons, WEAK[shell][1], 0)
    _, _, good = problem(shell, nucleons, None, 0)
    _, _, mixing = problem(shell, nucleons, None, 0, mix=True)
    pairs = [(*vac[0], *vac[1]), (*good[0], *good[1]), (*vac[1], *vac[0]), (*mixing[0], *mixing[1])]
    with PnampContext(*args, Mesh(2, 3, 3, 5), q2=q2, form="df64") as ctx:
        zd, st = ctx.batch(pairs)
        ctx.set_form("tc6")
        zt, sc = ctx.batch(pairs)
    assert st.max() == 0 and sc.max() == 0
    for a, b in zip(zt, zd):
        for io in range(NOBS):
            assert np.abs(a[:, io] - b[:, io]).max() <= (1e-6 if io == 6 else 1e-12) * np.abs(b[:, io]).max(), io


@pytest.mark.gpu
@pytest.mark.parametrize("gauge", [False, True])
@pytest.mark.parametrize("form", ["fp64", "df64"])
def test_weak_pairs_keep_the_species_split(form, gauge):
    """A conserving pair takes at most 0.6 of the time of a mixing pair of the same orders (NFOM^2 points
    of order n against species blocks), with and without the values of every gauge point."""
    import torch
    from sccm_gb300.pnamp import PnampContext
    ms = []
    for mix in (False, True):
        args, q2, vac = problem("pf", *WEAK["pf"], 0, mix=mix)
        with PnampContext(*args, Mesh(4, 8, 4, 5), q2=q2, form=form) as ctx:
            P = ctx.n_euler
            uv = torch.from_numpy(ctx.pack_pairs([(*vac[0], *vac[1])])).cuda()
            it = torch.tensor([(0, e) for e in range(P)], dtype=torch.int32, device="cuda")
            z = torch.zeros((1, NOBS, P, 2), dtype=torch.float64, device="cuda")
            st = torch.zeros((1, P), dtype=torch.int32, device="cuda")
            g = torch.zeros((1, P, 25, 4), dtype=torch.float64, device="cuda")
            stream = torch.cuda.current_stream().cuda_stream
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t = []
            for _ in range(4):
                a.record()
                ctx.batch_items_device(1, uv.data_ptr(), P, it.data_ptr(), z.data_ptr(), st.data_ptr(),
                                       g.data_ptr() if gauge else 0, stream)
                b.record()
                torch.cuda.synchronize()
                t.append(a.elapsed_time(b))
            ms.append(min(t[1:]))
    assert ms[0] <= 0.6 * ms[1], ms


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
def test_densities_of_a_batch_with_pairs_of_every_kind(form):
    """CTAs run pairs of different kinds side by side: every pair's densities are those of the pair
    alone (to the rounding of their order of summation)."""
    from sccm_gb300.pnamp import PnampContext
    args, q2, weak = problem("pf", *WEAK["pf"], 0)
    vac = [weak] + [problem("pf", (4, 4), gap, 0, mix=mix)[2] for gap, mix in ((None, False), (None, True), (0.2, True))]
    pairs = [(*v[i], *v[1 - i]) for v in vac for i in (0, 1)]
    with PnampContext(*args, Mesh(4, 8, 4, 3), q2=q2, form=form) as ctx:
        alone = [ctx.batch_densities([p]) for p in pairs]
        z, st, r1, r2 = ctx.batch_densities(pairs + pairs[::-1])
    assert st.max() == 0
    for k, p in enumerate(list(range(8)) + list(range(7, -1, -1))):
        za, _, r1a, r2a = alone[p]
        for got, ref in ((z[k], za[0]), (r1[k], r1a[0]), (r2[k], r2a[0])):
            assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max(), (k, p)


@pytest.mark.gpu
@pytest.mark.parametrize("shell,mix", [("sd", True), ("sd", False), ("pf", True), ("pf", False)])
def test_symmetric_errors_of_the_vacua_drop_out_of_the_norm(shell, mix):
    """V + d S U with S symmetric adds d S to V U^-1, whose skew part stays as it is, so the norm changes
    at second order only: d = 1e-9 leaves it to 1e-12 (upper triangles would show 1e-9)."""
    from sccm_gb300.pnamp import PnampContext
    args, q2, vac = problem(shell, (2, 2), None, 3, mix=mix)
    rng = np.random.default_rng(4)
    h = vac[0][0].shape[0] // 2
    same = np.kron(np.eye(2), np.ones((h, h))) if not mix else 1.0   # charge-conserving pairs stay so

    def moved(U, V):
        S = rng.standard_normal(U.shape) * same
        return U, V + 1e-9 * (S + S.T) @ U
    pairs = [(*vac[0], *vac[1]), (*moved(*vac[0]), *vac[1]), (*vac[0], *moved(*vac[1]))]
    with PnampContext(*args, Mesh(2, 4, 2, 3), q2=q2) as ctx:
        z, st = ctx.batch(pairs)
    assert st.max() == 0
    for k in (1, 2):
        assert np.abs(z[k][:, 0] - z[0][:, 0]).max() <= 1e-12 * np.abs(z[0][:, 0]).max(), k


@pytest.mark.gpu
def test_two_body_densities_of_half_filled_shells_in_double_float():
    """Bras with entries of Z0 = V0 U0^-1 from 10 to 19: kappa01 = Z0 + Z0 kappa10 Z0 cancels there, T22
    does not (4e-14 of the largest element over these pairs; 2e-13 by the single skew inverse)."""
    from sccm_gb300.pnamp import PnampContext
    sp = ModelSpace(SHELLS["pf"], 10, 10)
    rng = np.random.default_rng(7)
    spe = rng.uniform(-4.0, 0.0, len(sp.orbits))
    t1b = np.diag([spe[o] for o in sp.orbit]).astype(complex)
    recs, q2 = mscheme_pairs(sp), q2_operators(sp)
    v = [deformed_vacuum(sp, spe, 0.05 + 0.06 * k, 25.0, rng, q2=q2, gap=0.4) for k in range(8)]
    assert min(np.abs(V @ np.linalg.inv(U)).max() for U, V in v) > 8.0
    pairs = [(*v[i], *v[(i + d) % 8]) for d in (1, 3) for i in range(8)]
    vbar = 0.5 * np.random.default_rng(1).standard_normal(len(recs))
    r = []
    for form in ("fp64", "df64"):
        with PnampContext(sp, 0.0, t1b, recs, vbar, Mesh(1, 4, 1, 5), q2=q2, form=form) as ctx:
            r.append(ctx.batch_rho2b(pairs)[2])
    assert (np.abs(r[1] - r[0]).max(1) / np.abs(r[0]).max(1)).max() <= 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "df64"])
@pytest.mark.parametrize("shell,gap,mesh", [("sd", None, (1, 3, 2, 3)), ("sd", 0.2, (1, 3, 2, 3)), ("p2", None, (2, 2, 1, 5)),
                                            ("pf", None, (1, 2, 1, 4)), ("pf", 0.2, (1, 2, 1, 4))])
def test_values_of_every_gauge_point_match_the_oracle(shell, gap, mesh, form):
    """N and N (H/N) point by point, both kinds of charge-conserving pairs (FP64 rounding of the
    largest point, as for the sums)."""
    import torch
    from sccm_gb300.pnamp import PnampContext
    args, q2, vac = problem(shell, (2, 2), gap, 8)
    mesh, pair, log = Mesh(*mesh), (*vac[0], *vac[1]), []
    with PnampContext(*args, mesh, q2=q2, form=form) as ctx:
        P, G = ctx.n_euler, mesh.n_gauge
        uv = torch.from_numpy(ctx.pack_pairs([pair])).cuda()
        it = torch.tensor([(0, e) for e in range(P)], dtype=torch.int32, device="cuda")
        z = torch.zeros((1, NOBS, P, 2), dtype=torch.float64, device="cuda")
        st = torch.zeros((1, P), dtype=torch.int32, device="cuda")
        g = torch.full((1, P, G, 2, 2), 7.0, dtype=torch.float64, device="cuda")
        ctx.batch_items_device(1, uv.data_ptr(), P, it.data_ptr(), z.data_ptr(), st.data_ptr(), g.data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    g = torch.view_as_complex(g[0]).cpu().numpy()
    oracle(args, q2, mesh, pair, point_log=log)
    N = np.array([o[0] for *_, o in log]).reshape(P, G)
    NH = np.array([o[6] for *_, o in log]).reshape(P, G)
    assert st.max() == 0
    assert np.abs(g[:, :, 0] - N).max() <= 1e-10 * np.abs(N).max()
    assert np.abs(g[:, :, 0] * g[:, :, 1] - NH).max() <= 1e-9 * np.abs(NH).max()
