"""GPU tests of the star-state decision (the Riemann solve without the star state's sound speed)
where its bounds are not the usual ones: EOS tables whose heat capacity turns negative inside the
scanned temperatures or never is positive, tables of several range switches, and the FMA form
beyond the sonic point."""
import dataclasses

import numpy as np
import pytest

from common import FP64_TOL, eos9, gpu_zeros, oracle, params_for, rel_err, to_cpu, to_gpu
from particleclem_b200 import abi, hydro, workloads as wl

pytestmark = pytest.mark.gpu


def _table(name):
    """The 9-species table with one trait: cv of a species < 0 from 2200 K on (inside the
    states' temperatures), < 0 everywhere (its mass fraction of at most a third leaves the
    mixture's positive), or range switches spread over 1000-1400 K."""
    eos = eos9()
    lo, hi, tmid = np.array(eos.a_lo), np.array(eos.a_hi), np.array(eos.tmid, dtype=float)
    if name == "turns negative":
        hi[3, :5] = (1.0 + 11.0, -5e-3, 0.0, 0.0, 0.0)  # cv / R = 11 - 5e-3 T
    elif name == "never positive":
        lo[3, :5] = hi[3, :5] = (1.0 - 1e-3, 0.0, 0.0, 0.0, 0.0)
    elif name == "several switches":
        tmid = tmid + 50.0 * np.arange(9)
    return dataclasses.replace(eos, a_lo=lo, a_hi=hi, tmid=tmid)


def _patch(eos, mach, seed):
    nspec = eos.nspec
    p = wl.random_patch((9, 8, 7), seed, eos if nspec > 1 else None)
    u = p.fab.data
    u[abi.UMX:abi.UMZ + 1] *= mach
    u[abi.UEDEN] = u[abi.UEINT] + 0.5 * (u[abi.UMX:abi.UMZ + 1] ** 2).sum(0) / u[abi.URHO]
    hydro.init(0)
    hydro.set_eos(eos)
    oracle().set_eos(eos)
    return p


def _both(p, nspec, prec):
    dt = 0.3 * oracle().estdt(p.lo, p.hi, p.fab, p.dx)
    prm = params_for(p, dt, prec=prec, nspec=nspec)
    ref, _ = oracle().hydro_box(prm, p.lo, p.hi, p.fab)
    out = gpu_zeros(abi.nvar(nspec), p.lo, p.hi)
    hydro.hydro_box(prm, p.lo, p.hi, to_gpu(p.fab), out)
    return dt, ref, to_cpu(out)


@pytest.mark.parametrize("name", ["turns negative", "never positive", "several switches"])
@pytest.mark.parametrize("mach", [0.0, 1.0, 3.0, 8.0])
def test_fp64_source_equals_oracle_for_odd_eos_tables(name, mach):
    p = _patch(_table(name), mach, 21)
    _, ref, got = _both(p, 9, abi.PREC_FP64)
    assert np.isfinite(ref.data).all()
    np.testing.assert_array_equal(got, ref.data)


@pytest.mark.parametrize("nspec", [1, 9])
@pytest.mark.parametrize("mach", [0.0, 2.0, 6.0])
def test_fma_state_within_its_bound_beyond_the_sonic_point(nspec, mach):
    p = _patch(wl.GammaLaw() if nspec == 1 else eos9(), mach, 22)
    dt, ref, got = _both(p, nspec, abi.PREC_FP64_FAST)
    want = oracle().update_state(p.lo, p.hi, p.fab, ref, dt)
    have = oracle().update_state(p.lo, p.hi, p.fab, abi.Fab(got, tuple(p.lo)), dt)
    l1, linf = rel_err(have.view(p.lo, p.hi), want.view(p.lo, p.hi))
    assert l1 <= FP64_TOL and linf <= FP64_TOL, (l1, linf)
