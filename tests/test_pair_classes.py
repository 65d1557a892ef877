"""Charge-conserving pairs over the range of Pfaffian scales, gaps and fillings.

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
