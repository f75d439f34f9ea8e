"""GPU tests of the kernels' shortcuts where they can go wrong: quotients by a shared
denominator at the ends of the exponent range, the star-state decision around and beyond the
sonic point, march lengths, overlapped launches, and the ghost fill and timestep reduction at
odd sizes. The plain FP64 form is compared bit for bit with the CPU oracle."""
import numpy as np
import pytest

from common import MIXED_TOL, eos9, gpu_zeros, oracle, params_for, rel_err, to_cpu, to_gpu
from particleclem_b200 import abi, hydro, thermo, workloads as wl

pytestmark = pytest.mark.gpu
FORMS = [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED]


def _eos(nspec):
    eos = wl.GammaLaw() if nspec == 1 else eos9()
    hydro.init(0)
    hydro.set_eos(eos)
    oracle().set_eos(eos)
    return eos


def _patch(edges, seed, nspec, mach=1.0):
    """random_patch with its velocities multiplied by mach; sets the EOS of its species count."""
    p = wl.random_patch(edges, seed, _eos(nspec))
    u = p.fab.data
    u[abi.UMX:abi.UMZ + 1] *= mach
    u[abi.UEDEN] = u[abi.UEINT] + 0.5 * (u[abi.UMX:abi.UMZ + 1] ** 2).sum(0) / u[abi.URHO]
    return p


def _run(p, nspec, prec, dx=None, **kw):
    _eos(nspec)
    dx = dx or p.dx
    dt = 0.3 * oracle().estdt(p.lo, p.hi, p.fab, dx)
    prm = params_for(p, dt, prec=prec, nspec=nspec, **kw)
    prm.dx[:] = list(dx)
    ref, flx = oracle().hydro_box(prm, p.lo, p.hi, p.fab)
    out = gpu_zeros(abi.nvar(nspec), p.lo, p.hi)
    got_flx = [gpu_zeros(abi.nvar(nspec), *abi.nodes(p.lo, p.hi, d)) for d in range(3)]
    hydro.hydro_box(prm, p.lo, p.hi, to_gpu(p.fab), out, got_flx)
    return dt, ref, flx, to_cpu(out), [to_cpu(f) for f in got_flx]


@pytest.mark.parametrize("nspec", [1, 9])
@pytest.mark.parametrize("scale", [1e-55, 1e-40, 1.0, 1e40, 1e55])
def test_fp64_source_equals_oracle_for_cell_sizes_across_the_exponent_range(nspec, scale):
    """The cell volume (scale^3) divides every flux sum: inside 2^-500..2^500 by its shared
    reciprocal, outside plainly."""
    p = _patch((7, 6, 5), 3, nspec)
    _, ref, flx, got, got_flx = _run(p, nspec, abi.PREC_FP64, dx=tuple(scale * d for d in p.dx))
    np.testing.assert_array_equal(got, ref.data)
    for d in range(3):
        np.testing.assert_array_equal(got_flx[d], flx[d].data)


@pytest.mark.parametrize("value", [0.0, -0.0, 5e-324, 1e-310, 1e-200, 1e-12, 1e160, np.inf, np.nan])
def test_ctoprim_mass_fractions_equal_oracle_for_odd_partial_densities(value):
    p = _patch((6, 5, 4), 4, 9)
    p.fab.data[abi.UFS + 2, 3:6, 2:5, 1:7] = value
    lo, hi = abi.grow(p.lo, p.hi, 4)
    q_ref, qa_ref = oracle().ctoprim(lo, hi, p.fab)
    q, qa = gpu_zeros(abi.qvar(9), lo, hi), gpu_zeros(abi.NQAUX, lo, hi)
    hydro.ctoprim(params_for(p, 0.0, nspec=9), lo, hi, to_gpu(p.fab), q, qa)
    got, want = to_cpu(q), q_ref.data
    np.testing.assert_array_equal(got, want)
    fine = ~np.isnan(want)
    np.testing.assert_array_equal(np.signbit(got)[fine], np.signbit(want)[fine])
    np.testing.assert_array_equal(to_cpu(qa), qa_ref.data)


@pytest.mark.parametrize("nspec", [1, 9])
@pytest.mark.parametrize("ppm", [0, 1])
@pytest.mark.parametrize("mach", [0.0, 2.0, 6.0, 20.0])
def test_fp64_source_equals_oracle_around_and_beyond_the_sonic_point(nspec, ppm, mach):
    p = _patch((9, 8, 7), 5, nspec, mach)
    _, ref, flx, got, got_flx = _run(p, nspec, abi.PREC_FP64, ppm_type=ppm)
    np.testing.assert_array_equal(got, ref.data)
    for d in range(3):
        np.testing.assert_array_equal(got_flx[d], flx[d].data)


@pytest.mark.parametrize("nspec", [1, 9])
@pytest.mark.parametrize("mach", [0.0, 4.0])
def test_mixed_state_within_its_bound_beyond_the_sonic_point(nspec, mach):
    p = _patch((9, 8, 7), 6, nspec, mach)
    dt, ref, _, got, _ = _run(p, nspec, abi.PREC_MIXED)
    want = oracle().update_state(p.lo, p.hi, p.fab, ref, dt)
    have = oracle().update_state(p.lo, p.hi, p.fab, abi.Fab(got, tuple(p.lo)), dt)
    l1, _ = rel_err(have.view(p.lo, p.hi), want.view(p.lo, p.hi))
    assert l1 <= MIXED_TOL, l1


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("nspec", [1, 9])
def test_source_does_not_depend_on_the_march_length(prec, nspec):
    """A box alone (short marches), and beside boxes that take the call past the cell counts
    where the marches lengthen."""
    _eos(nspec)
    small = _patch((13, 11, 9), 7, nspec)
    outs = []
    for n in (0, 44, 52):
        patches = [small] + ([wl.random_patch((n, n, n), 8, _eos(nspec))] if n else [])
        boxes, res = [], gpu_zeros(abi.nvar(nspec), small.lo, small.hi)
        for m, p in enumerate(patches):
            dt = 0.3 * oracle().estdt(p.lo, p.hi, p.fab, p.dx)
            out = res if m == 0 else gpu_zeros(abi.nvar(nspec), p.lo, p.hi)
            boxes.append(hydro.make_box(p.lo, p.hi, to_gpu(p.fab), out, p.dx, dt))
        hydro.hydro_boxes(params_for(small, 0.0, prec=prec, nspec=nspec), boxes)
        outs.append(to_cpu(res))
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("nspec", [1, 9])
def test_overlapped_launches_equal_stages_run_one_by_one(prec, nspec):
    """The launches of one call may overlap; each stage alone, waited for, does not."""
    import torch

    p = _patch((17, 9, 12), 9, nspec)
    uin, out = to_gpu(p.fab), gpu_zeros(abi.nvar(nspec), p.lo, p.hi)
    plan = hydro.Plan(params_for(p, 0.0, prec=prec, nspec=nspec),
                      [hydro.make_box(p.lo, p.hi, uin, out, p.dx, 0.0)])
    dt0 = oracle().estdt(p.lo, p.hi, p.fab, p.dx)
    for cfl in np.linspace(0.05, 0.5, 12):
        dt = torch.tensor([cfl * dt0], dtype=torch.float64, device="cuda")
        for st in range(7):
            plan.stages(st, st, dt)
            torch.cuda.synchronize()
        want = to_cpu(out)
        out.data.zero_()
        plan.hydro(dt)
        np.testing.assert_array_equal(to_cpu(out), want)


@pytest.mark.parametrize("ncomp", [1, 7, 8, 9, 28])
@pytest.mark.parametrize("periodic", [(True, False, True), (False, True, False)])
def test_ghost_fill_equals_the_numpy_fill(ncomp, periodic):
    rng = np.random.default_rng(ncomp)
    u = rng.standard_normal((ncomp, 5 + 8, 4 + 8, 6 + 8))
    want = u.copy()
    wl.fill_ghosts(want, periodic)
    fab = to_gpu(abi.Fab(u, (-4, -4, -4)))
    hydro.fill_ghosts(fab, (0, 0, 0), (5, 3, 4), periodic)
    np.testing.assert_array_equal(to_cpu(fab), want)


@pytest.mark.parametrize("edges", [(1, 1, 1), (33, 31, 4), (64, 64, 33), (160, 128, 96)])
def test_timestep_reduction_equals_the_oracle(edges):
    """From one block's minimum to more minima than one block of the final reduction takes."""
    import torch

    p = _patch(edges, 10, 1)
    dt = torch.zeros(1, dtype=torch.float64, device="cuda")
    hydro.estdt(1, [hydro.make_box(p.lo, p.hi, to_gpu(p.fab), None, p.dx, 0.0)], 0.4, dt)
    assert dt.item() == 0.4 * oracle().estdt(p.lo, p.hi, p.fab, p.dx)


@pytest.mark.parametrize("nspec", [2, 3])
@pytest.mark.parametrize("edges", [(35, 34, 33), (44, 41, 39)])
def test_few_species_equal_oracle_on_both_sides_of_the_launch_size_rule(nspec, edges):
    """Launches of up to 1184 blocks (128 faces each) and larger ones run the FP64
    stages of 2 to 5 species at different register caps."""
    if nspec not in hydro.species_counts():
        pytest.skip(f"library built without {nspec} species")
    eos = thermo.standin_mixture(nspec)
    hydro.init(0)
    hydro.set_eos(eos)
    oracle().set_eos(eos)
    p = wl.random_patch(edges, 17, eos)
    prm = params_for(p, 0.3 * oracle().estdt(p.lo, p.hi, p.fab, p.dx), prec=abi.PREC_FP64, nspec=nspec)
    ref, _ = oracle().hydro_box(prm, p.lo, p.hi, p.fab)
    out = gpu_zeros(abi.nvar(nspec), p.lo, p.hi)
    hydro.hydro_box(prm, p.lo, p.hi, to_gpu(p.fab), out)
    np.testing.assert_array_equal(to_cpu(out), ref.data)
